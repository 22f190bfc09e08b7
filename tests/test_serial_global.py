"""Serial bodies larger than a pack, replayed from global memory: carried and
plain records, whole updates and link passes.  Bit-exact against the oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


def _chain(kind, n):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    pos = np.stack([3.0 + 0.5 * (i % 700), 5.0 + 2.0 * (i // 700) + rng.uniform(0.0, 0.5, n)], 1)
    a, b = i[:-1], i[1:]
    if kind == "doubled":  # consecutive links share both particles: records without marks
        a, b = np.repeat(a, 2), np.repeat(b, 2)
    elif kind == "braced":
        a, b = np.concatenate([a, i[:-2]]), np.concatenate([b, i[2:]])
    elif kind == "ring":
        rim = i[:-1]
        a = np.concatenate([rim, rim])
        b = np.concatenate([(rim + 1) % (n - 1), np.full(n - 1, n - 1)])
    return (pos.astype(np.float32), np.minimum(a, b).astype(np.uint64),
            np.maximum(a, b).astype(np.uint64))


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("kind", ["rope", "doubled", "braced", "ring"])
def test_chains_past_a_pack(gpu, kind, collide):
    from bendy2d_gb300 import scenes
    from oracle import load_scene
    sc = scenes._assemble(kind, [_chain(kind, 13001)], bounds=(0.0, 0.0, 400.0, 400.0), sub_steps=2,
                          link_iters=3, collide=collide)
    sc.prev = scenes._velocity_prev(sc.pos, np.random.default_rng(1), 0.5, sc.dt / 2)
    sc.stiff = np.random.default_rng(2).uniform(0.5, 1.0, len(sc.la)).astype(np.float32)
    s, o = sc.to_solver(), load_scene(sc)
    s.set_tuning(serial_width=1e9)
    assert s.plan_stats()["serial_bodies"] == 1
    s.set_profiling(True)
    s.update(sc.dt)
    assert f"exec_serial_{'links' if collide else 'full'}" in s.profile()
    s.set_profiling(False)
    s.update(sc.dt)
    for _ in range(2):
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), kind)
    s.close()

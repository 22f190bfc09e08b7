"""link_iters = 0: the links are never applied, whatever executor a body runs
on; bounds, integration and collisions go on.  Bit-exact against the oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu

SERIAL = {"serial_width": 1e9}


def _rope(n, y):
    rng = np.random.default_rng(n)
    pos = np.stack([3.0 + 0.5 * np.arange(n), y + rng.uniform(0.0, 2.0, n)], 1).astype(np.float32)
    a = np.arange(n - 1, dtype=np.uint64)
    return pos, a, a + np.uint64(1)


def _ring(n, y):
    """A rim and its spokes to a hub: two chains in the serial executor."""
    pos, _, _ = _rope(n, y)
    rim, hub = np.arange(n - 1), np.full(n - 1, n - 1)
    a, b = np.concatenate([rim, rim]), np.concatenate([(rim + 1) % (n - 1), hub])
    return pos, np.minimum(a, b).astype(np.uint64), np.maximum(a, b).astype(np.uint64)


def _check(bodies, sub_steps, collide, tuning, case="", box=400.0, link_iters=0):
    from bendy2d_gb300 import scenes
    from oracle import load_scene
    sc = scenes._assemble("no links", bodies, bounds=(0.0, 0.0, box, box), sub_steps=sub_steps,
                          link_iters=link_iters, collide=collide)
    sc.prev = scenes._velocity_prev(sc.pos, np.random.default_rng(1), 0.5, sc.dt / sub_steps)
    if case == "replayed":  # a coordinate -0 keeps a body off the fused solve
        sc.pos[::7] = (-0.0, -0.0)
    s, o = sc.to_solver(), load_scene(sc)
    s.set_tuning(**tuning)
    for _ in range(2):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), f"{tuning} {case}")
    s.close()


@pytest.mark.parametrize("case", ["", "replayed"])
@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("sub_steps", [1, 2, 3, 8])
@pytest.mark.parametrize("tuning", [{}, SERIAL, {**SERIAL, "stage_frac": 0.0}, {"serial_width": 0.0},
                                    {"serial_width": 0.0, "smem_max": 1024}])
def test_chains(gpu, tuning, sub_steps, collide, case):
    bodies = [f(n, 5.0 + 8.0 * k) for k, (f, n) in enumerate(
        [(_rope, 3), (_rope, 50), (_rope, 300), (_ring, 12), (_ring, 41), (_ring, 150)])]
    _check(bodies, sub_steps, collide, tuning, case)


@pytest.mark.parametrize("collide", [0, 1])
def test_chain_past_a_pack(gpu, collide):
    _check([_rope(14000, 5.0)], 2, collide, SERIAL, box=8000.0)


def test_worlds_of_one_pack_with_and_without_link_iterations(gpu):
    """Bodies of one pack, some of worlds with links and some without."""
    from bendy2d_gb300 import Batch, scenes
    from oracle import load_scene
    scs = [scenes._assemble("w", [_ring(n, 5.0)], bounds=(0.0, 0.0, 400.0, 400.0),
                            sub_steps=1 + n % 3, link_iters=it)
           for n, it in ((41, 0), (30, 2), (55, 0), (41, 1))]
    solvers, oracles = [sc.to_solver() for sc in scs], [load_scene(sc) for sc in scs]
    b = Batch(solvers)
    b.set_tuning(**SERIAL)
    for _ in range(2):
        b.update(scs[0].dt)
        for o, sc in zip(oracles, scs):
            assert o.update(sc.dt) == 0
    for s, o in zip(solvers, oracles):
        assert_same_state(solver_state(s), oracle_state(o))
    b.close()

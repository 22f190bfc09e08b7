"""Particles without links, in fewer and in more bodies than the GPU has
multiprocessors, alone and beside cloths.  Bit-exact against the oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("free_chunk", [256, 257, 700, 2048])
@pytest.mark.parametrize("n,cloths", [(1000, 1), (60001, 0), (250003, 0), (250003, 3)])
def test_free_particles(gpu, n, cloths, free_chunk):
    from bendy2d_gb300 import scenes
    from oracle import load_scene
    rng = np.random.default_rng(n)
    none = np.zeros(0, np.uint64)
    bodies = [scenes.grid_body(20, 17, (5.0 + 30.0 * k, 5.0), 1.0, 0.01, rng) for k in range(cloths)]
    bodies.append((rng.uniform(1.0, 399.0, (n, 2)).astype(np.float32), none, none))
    sc = scenes._assemble("free", bodies, bounds=(0.0, 0.0, 400.0, 400.0), sub_steps=3, link_iters=2)
    sc.prev = scenes._velocity_prev(sc.pos, rng, 2.0, sc.dt / 3)
    s, o = sc.to_solver(), load_scene(sc)
    s.set_tuning(free_chunk=free_chunk)
    for _ in range(2):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), f"{n} particles in bodies of {free_chunk}")
    s.close()


def test_batch_of_more_bodies_than_sms(gpu):
    from bendy2d_gb300 import Batch, scenes
    from oracle import load_scene
    none = np.zeros(0, np.uint64)
    scs = []
    for k in range(60):
        rng = np.random.default_rng(k)
        sc = scenes._assemble("w", [(rng.uniform(1.0, 99.0, (5000 + k, 2)).astype(np.float32), none, none)],
                              bounds=(0.0, 0.0, 100.0, 100.0), sub_steps=1 + k % 3, link_iters=1)
        sc.prev = scenes._velocity_prev(sc.pos, rng, 2.0, sc.dt)
        scs.append(sc)
    solvers, oracles = [sc.to_solver() for sc in scs], [load_scene(sc) for sc in scs]
    b = Batch(solvers)
    for _ in range(2):
        b.update(scs[0].dt)
        for o, sc in zip(oracles, scs):
            assert o.update(sc.dt) == 0
    for s, o in zip(solvers, oracles):
        assert_same_state(solver_state(s), oracle_state(o))
    b.close()

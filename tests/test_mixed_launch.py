"""Bodies of every group size in one launch, one body per CTA whose idle warps
leave: resident and streamed schedules, whole updates and link passes, unit
and other stiffnesses, a body that takes the general solve, as many bodies as
SMs and one more.  Bit-exact against the oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu

SIZES = [(40, 30), (2, 2), (8, 8), (25, 13), (3, 60), (32, 32), (5, 4), (16, 9)]


def _scene(sizes, collide, stiff=None, neg0=False, link_iters=2):
    from bendy2d_gb300 import scenes
    rng = np.random.default_rng(5)
    bodies = [scenes.grid_body(w, h, (3.0 + 45.0 * (k % 20), 3.0 + 65.0 * (k // 20)), 1.0, 0.01, rng)
              for k, (w, h) in enumerate(sizes)]
    sc = scenes._assemble("mixed", bodies, bounds=(0.0, 0.0, 1000.0, 1000.0), sub_steps=2,
                          link_iters=link_iters, collide=collide)
    if neg0:  # in the second body
        sc.pos[len(bodies[0][0]), 0] = -0.0
    sc.prev = scenes._velocity_prev(sc.pos, np.random.default_rng(2), 0.5, sc.dt / 2)
    if stiff is not None:
        sc.stiff = np.where(np.arange(len(sc.la)) % 3 == 0, np.float32(stiff), np.float32(1.0))
    return sc


def _check(sc, what, launches=None, tuning=None):
    from oracle import load_scene
    s = sc.to_solver()
    s.set_tuning(serial_width=0.0, **(tuning or {}))
    o = load_scene(sc)
    for _ in range(2):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    if launches is not None:
        assert s.launch_count() == launches
    assert_same_state(solver_state(s), oracle_state(o), what)
    s.close()


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("stiff,neg0", [(None, False), (0.4, False), (None, True)])
def test_every_group_size_in_one_launch(gpu, resident, collide, stiff, neg0):
    _check(_scene(SIZES, collide, stiff, neg0), f"resident {resident} collide {collide}",
           launches=1 if not collide and not resident else None, tuning={"resident": resident})


@pytest.mark.parametrize("collide", [0, 1])
def test_as_many_bodies_as_sms_and_one_more(gpu, collide):
    import torch
    n = torch.cuda.get_device_properties(0).multi_processor_count
    for k in (n, n + 1):
        sizes = [SIZES[i % len(SIZES)][::-1] if i % 7 else (20, 3) for i in range(k)]
        _check(_scene([(min(w, 20), min(h, 20)) for w, h in sizes], collide, link_iters=1),
               f"{k} bodies", tuning={"resident": 0})

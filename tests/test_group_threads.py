"""Group sizes at the ends of the tunables' ranges: many one-warp groups in a
CTA, and the largest groups, for whole updates and for link passes.  Bit-exact
against the oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


def _scene(n_bodies, w, h, collide):
    from bendy2d_gb300 import scenes
    rng = np.random.default_rng(3)
    gap = 1.6 * max(w, h)
    bodies = [scenes.grid_body(w, h, (5.0 + gap * (k % 30), 5.0 + gap * (k // 30)), 1.0, 0.01, rng)
              for k in range(n_bodies)]
    sc = scenes._assemble("groups", bodies, bounds=(0.0, 0.0, 400.0, 400.0), sub_steps=2,
                          link_iters=2, collide=collide)
    sc.prev = scenes._velocity_prev(sc.pos, rng, 0.5, sc.dt / 2)
    return sc


def _check(sc, tuning):
    from oracle import load_scene
    s, o = sc.to_solver(), load_scene(sc)
    s.set_tuning(**tuning)
    for _ in range(2):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), str(tuning))
    s.close()


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("warp_groups", [16, 17, 24, 32])
def test_one_warp_groups_of_more_bodies_than_sms(gpu, warp_groups, collide):
    _check(_scene(500, 3, 4, collide), {"warp_groups": warp_groups, "pack_np": 1, "serial_width": 0.0,
                                        "t_max": 32})


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("smem_max", [1024, 200 * 1024])
@pytest.mark.parametrize("t", [{"t_max": 1024}, {"t_min": 1024, "t_max": 1024},
                               {"t_max": 1024, "width_per_thread": 0.01}])
def test_largest_groups(gpu, t, smem_max, collide):
    _check(_scene(2, 40, 30, collide), {**t, "smem_max": smem_max, "large_max": 0})

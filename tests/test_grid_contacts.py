"""Particle contacts over the collision grid, both forms of the collide pass
on both grids: cells from empty to more entries than a bucket's slots, more
contacts than a lane keeps, coincident particles, differences too small for
the fused solve, every particle count around a warp's and a chunk's edges.
Bit-exact against the oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu

FORMS = [{"collide_thread_min": 1 << 30}, {"collide_thread_min": 0},
         {"collide_thread_min": 1 << 30, "grid_slot_max": 0},
         {"collide_thread_min": 0, "grid_slot_max": 0}]


def _check(pos, box, tuning, what, cell=1.0, steps=2, sub_steps=3):
    from bendy2d_gb300 import scenes
    from oracle import load_scene
    none = np.zeros(0, np.uint64)
    sc = scenes._assemble("grains", [(np.asarray(pos, np.float32), none, none)],
                          bounds=(0.0, 0.0, box, box), sub_steps=sub_steps, collide=1)
    sc.cell = cell
    sc.prev = scenes._velocity_prev(sc.pos, np.random.default_rng(2), 0.5, sc.dt / sub_steps)
    s = sc.to_solver()
    s.set_tuning(**tuning)
    o = load_scene(sc)
    for _ in range(steps):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), what)
    s.close()


@pytest.mark.parametrize("tuning", FORMS)
@pytest.mark.parametrize("n,box", [(1, 20.0), (9, 4.0), (10, 40.0), (11, 3.0), (33, 6.0),
                                   (319, 30.0), (320, 12.0), (321, 18.0), (700, 9.0)])
def test_loose_particles_of_any_density(gpu, n, box, tuning):
    pos = np.random.default_rng(n).uniform(0.0, box, (n, 2))
    _check(pos, box, tuning, f"{n} in {box}")


@pytest.mark.parametrize("tuning", FORMS)
def test_coincident_and_nearly_coincident_particles(gpu, tuning):
    rng = np.random.default_rng(4)
    base = rng.uniform(2.0, 28.0, (60, 2)).astype(np.float32)
    near = base.copy()
    near[:20, 0] = np.nextafter(near[:20, 0], np.float32(100.0))
    tiny = np.array([[0.0, 0.0], [1e-20, 0.0], [0.0, 1e-30], [1e-16, 1e-17], [0.25, 1e-25]])
    _check(np.vstack([base, near, base[30:], tiny]), 30.0, tuning, "coincident")


@pytest.mark.parametrize("tuning", FORMS)
def test_cell_that_needs_a_division(gpu, tuning):
    pos = np.random.default_rng(6).uniform(0.0, 20.0, (500, 2))
    _check(pos, 20.0, tuning, "cell 1.3", cell=1.3)

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


def _check(pos, box, tuning, what, cell=1.0, steps=2, sub_steps=3, circles=(), polygons=()):
    from bendy2d_gb300 import scenes
    from oracle import load_scene
    none = np.zeros(0, np.uint64)
    sc = scenes._assemble("grains", [(np.asarray(pos, np.float32), none, none)],
                          bounds=(0.0, 0.0, box, box), sub_steps=sub_steps,
                          collide=7 if circles or polygons else 1, circles=list(circles),
                          polygons=list(polygons))
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


def _bodies(rng, n_circles, n_polys, box):
    from bendy2d_gb300 import scenes
    circles = [scenes._circle(rng.uniform(0, box, 2), rng.uniform(1, 4), k % 2 == 0)
               for k in range(n_circles)]
    polys = [{"points": scenes.convex_polygon(rng, rng.uniform(3, box - 3, 2), rng.uniform(2, 5),
                                              4 + k % 5), "static": k % 3 == 0}
             for k in range(n_polys)]
    return circles, polys


@pytest.mark.parametrize("tuning", FORMS)
@pytest.mark.parametrize("n_circles,n_polys", [(1, 0), (0, 1), (31, 2), (33, 31), (40, 30), (70, 0)])
def test_particles_among_circles_and_polygons(gpu, n_circles, n_polys, tuning):
    """Particles pushed from one body into the next, more bodies than lanes."""
    rng = np.random.default_rng(n_circles + n_polys)
    circles, polys = _bodies(rng, n_circles, n_polys, 30.0)
    _check(rng.uniform(0.0, 30.0, (400, 2)), 30.0, tuning, "among bodies", circles=circles,
           polygons=polys)


@pytest.mark.parametrize("slots", [0, 1 << 20])
@pytest.mark.parametrize("bodies", [False, True])
def test_more_ctas_than_five_an_sm(gpu, slots, bodies):
    import torch
    n = torch.cuda.get_device_properties(0).multi_processor_count * 5 * 80 + 700
    rng = np.random.default_rng(3)
    circles, polys = _bodies(rng, 20, 5, 300.0) if bodies else ((), ())
    _check(rng.uniform(0.0, 300.0, (n, 2)), 300.0,
           {"collide_thread_min": 1 << 30, "grid_slot_max": slots}, "six an SM", steps=1,
           sub_steps=2, circles=circles, polygons=polys)

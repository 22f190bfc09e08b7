"""Bodies over one CTA's shared memory, run by a cluster whose CTAs pass
particles to one another: 2 to 8 CTAs, spatial and scattered particle orders,
whole-update and link-pass schedules, operands outside the fused solve's
range, more bodies than the GPU holds at a time.  Bit-exact against the
oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


def _cloth(w, h, origin=(5.0, 5.0), seed=1, scatter=False):
    from bendy2d_gb300 import scenes
    pos, a, b = scenes.grid_body(w, h, origin, 1.0, 0.01, np.random.default_rng(seed))
    if scatter:  # the same cloth with its particles numbered at random
        to = np.random.default_rng(9).permutation(len(pos))
        out = np.empty_like(pos)
        out[to] = pos
        x, y = to[a.astype(np.int64)], to[b.astype(np.int64)]
        pos, a, b = out, np.minimum(x, y).astype(np.uint64), np.maximum(x, y).astype(np.uint64)
    return pos, a, b


def _scene(bodies, collide=0, sub_steps=2, link_iters=2, stiff=None, box=300.0):
    from bendy2d_gb300 import scenes
    sc = scenes._assemble("large", bodies, bounds=(0.0, 0.0, box, box), sub_steps=sub_steps,
                          link_iters=link_iters, collide=collide)
    sc.prev = scenes._velocity_prev(sc.pos, np.random.default_rng(2), 0.5, sc.dt / sub_steps)
    if stiff is not None:
        sc.stiff = np.full(len(sc.la), stiff, np.float32)
    return sc


def _check(sc, what, steps=2, tuning=None):
    from oracle import load_scene
    s = sc.to_solver()
    if tuning:
        s.set_tuning(**tuning)
    st = s.plan_stats()
    assert st["large_bodies"] > 0 and st["global_bodies"] == 0
    o = load_scene(sc, link_order=s.link_order() if sc.mode else None)
    for _ in range(steps):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), what)
    s.close()


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("large_max", [2, 3, 5, 8])
@pytest.mark.parametrize("w,h,scatter", [(40, 33, False), (33, 40, True), (3, 90, False)])
def test_small_bodies_pushed_to_the_cluster(gpu, w, h, scatter, large_max, collide):
    sc = _scene([_cloth(w, h, scatter=scatter)], collide, sub_steps=3, link_iters=3)
    _check(sc, f"{w}x{h} on {large_max}", tuning={"smem_max": 1024, "large_max": large_max,
                                                  "serial_width": 0.0})


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("stiff", [None, 0.6])
def test_large_cloths(gpu, stiff, mode):
    sc = _scene([_cloth(110, 64), _cloth(80, 75, (150.0, 150.0))], sub_steps=4, link_iters=4,
                stiff=stiff)
    sc.mode = mode
    _check(sc, "two large cloths")


@pytest.mark.parametrize("case", ["tiny", "negative_zero", "coincident", "huge_rest", "far"])
@pytest.mark.parametrize("collide", [0, 1])
def test_operands_out_of_range_run_again(gpu, case, collide):
    pos, a, b = _cloth(30, 30)
    if case == "tiny":
        pos[400:406, 0] = [0.0, 1e-20, 3e-18, 1e-40, 4e-16, 2e-13]
    elif case == "negative_zero":
        pos[7] = (-0.0, -0.0)
    elif case == "coincident":
        pos[500] = pos[501]
    elif case == "far":
        pos[3] = (3e19, 2e19)
    sc = _scene([(pos, a, b)], collide)
    if case == "huge_rest":
        sc.rest[1000] = np.float32(3e38)
    _check(sc, case, tuning={"smem_max": 1024})


def test_more_clusters_than_the_gpu_holds(gpu):
    bodies = [_cloth(24 + k % 3, 20, (5.0 + 28.0 * (k % 10), 5.0 + 25.0 * (k // 10)), seed=k)
              for k in range(80)]
    _check(_scene(bodies), "80 bodies", tuning={"smem_max": 1024, "pack_np": 1})


@pytest.mark.parametrize("w,h,mode", [(100, 100, 0), (72, 80, 1)])
def test_levels_of_more_links_than_threads(gpu, w, h, mode):
    """The widest CTA's levels take two rounds of fewer threads."""
    sc = _scene([_cloth(w, h)], sub_steps=2, link_iters=4)
    sc.mode = mode
    _check(sc, f"{w}x{h} mode {mode}", steps=1)

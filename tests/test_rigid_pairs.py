"""Circle and polygon pairs: overlapping and separate bodies, polygons up to
and past the size whose edges are listed, more stages than a CTA has threads,
points past a warp's lanes, axis-aligned neighbours, coordinates that overflow
a product, whole updates and the sub-step pipeline.  Bit-exact against the
oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


def _polygon(rng, center, radius, n):
    from bendy2d_gb300 import scenes
    return {"points": scenes.convex_polygon(rng, center, radius, n), "static": False}


def _check(circles, polys, box, what, collide=0, sub_steps=3, steps=3, link_iters=1):
    from bendy2d_gb300 import scenes
    from oracle import load_scene
    bodies = []
    if collide:
        none = np.zeros(0, np.uint64)
        bodies = [(np.random.default_rng(3).uniform(0, box, (50, 2)), none, none)]
    sc = scenes._assemble("pairs", bodies, circles=circles, polygons=polys,
                          bounds=(0.0, 0.0, box, box), sub_steps=sub_steps,
                          link_iters=link_iters, collide=collide)
    s, o = sc.to_solver(), load_scene(sc)
    for _ in range(steps):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), what)
    s.close()


@pytest.mark.parametrize("collide", [0, 7])
@pytest.mark.parametrize("n,spread", [(2, 0.5), (5, 0.6), (17, 0.8), (24, 2.0), (40, 0.9)])
def test_polygons_from_piled_up_to_apart(gpu, n, spread, collide):
    rng = np.random.default_rng(n)
    side = int(np.ceil(np.sqrt(n)))
    polys = [_polygon(rng, (12.0 + 16.0 * spread * (k % side), 12.0 + 16.0 * spread * (k // side)),
                      rng.uniform(5.0, 10.0), 3 + k % 7) for k in range(n)]
    _check([], polys, 40.0 + 16.0 * spread * side, f"{n} polygons", collide)


@pytest.mark.parametrize("sizes", [(63, 64, 5), (64, 40, 33), (65, 4, 4), (31, 32, 33, 6),
                                   (130, 90), (4, 200, 3)])
def test_polygons_around_the_listed_size(gpu, sizes):
    rng = np.random.default_rng(sum(sizes))
    polys = [_polygon(rng, (30.0 + 18.0 * (k % 2), 30.0 + 14.0 * (k // 2)), 11.0, n)
             for k, n in enumerate(sizes)]
    _check([], polys, 100.0, f"vertices {sizes}", steps=2)


def test_axis_aligned_neighbours(gpu):
    """Edges on common lines, touching and apart: quotients of exact zeros."""
    square = np.array([[0, 0], [4, 0], [4, 4], [0, 4]], np.float32)
    polys = [{"points": square + np.float32([x, y]), "static": False}
             for x, y in [(10, 10), (14, 10), (18, 10), (30, 10), (10, 14), (12, 16), (40, 30)]]
    _check([], polys, 60.0, "squares")


@pytest.mark.parametrize("scale", [1e-12, 1e12, 1e18])
def test_extreme_coordinates(gpu, scale):
    rng = np.random.default_rng(8)
    polys = [{"points": (_polygon(rng, (20.0 + 12.0 * k, 20.0), 8.0, 5)["points"] * scale)
              .astype(np.float32), "static": False} for k in range(4)]
    _check([], polys, 100.0 * scale, f"scale {scale}", sub_steps=2, steps=1)


@pytest.mark.parametrize("n,box", [(2, 8.0), (23, 30.0), (24, 60.0), (46, 40.0), (60, 120.0)])
def test_circles_from_piled_up_to_apart(gpu, n, box):
    from bendy2d_gb300 import scenes
    rng = np.random.default_rng(n)
    circles = [scenes._circle(rng.uniform(0, box, 2), rng.uniform(1, 5), k % 4 == 0)
               for k in range(n)]
    _check(circles, [_polygon(rng, (5.0, 5.0), 3.0, 4)], box, f"{n} circles", link_iters=3)

"""The shared-memory link executor against the oracle where its fused link
solve could go wrong: operands outside the range it counts on (the body then
runs again with the IEEE form), quotients at the exceptional significands of
the fused division, rounds narrower and wider than the group, schedules held
whole and streamed.  Bit-exact (NaN-aware), as every parity test."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


def _scene(bodies, collide, sub_steps=2, link_iters=3, stiff=None, rest=None, box=200.0):
    from bendy2d_gb300 import scenes
    sc = scenes._assemble("links", bodies, bounds=(-box / 2, -box / 2, box, box),
                          sub_steps=sub_steps, link_iters=link_iters, collide=collide)
    rng = np.random.default_rng(3)
    sc.prev = scenes._velocity_prev(sc.pos, rng, 0.5, sc.dt / sc.sub_steps)
    if stiff is not None:
        sc.stiff = np.full(len(sc.la), stiff, np.float32)
    if rest is not None:
        sc.rest[:: 7] = rest
    return sc


def _grid(w, h, origin=(-20.0, -10.0), jitter=0.01, seed=1):
    from bendy2d_gb300 import scenes
    return scenes.grid_body(w, h, origin, 1.0, jitter, np.random.default_rng(seed))


def _check(sc, what, steps=2, tuning=None):
    from oracle import load_scene
    s = sc.to_solver()
    if tuning:
        s.set_tuning(**tuning)
    order = s.link_order() if sc.mode else None
    o = load_scene(sc, link_order=order)
    for _ in range(steps):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), what)
    s.close()


def _near_zero(body):
    """Columns of the grid at x within 1e-12 of zero, some of them -0, some
    subnormal: differences below 2^-50 in every link along a column."""
    pos, a, b = body
    pos = pos.copy()
    tiny = np.array([0.0, -0.0, 1e-20, -3e-18, 1e-40, 4e-16, 2e-13], np.float32)
    col = np.abs(pos[:, 0] - pos[:, 0].min()) < 0.5
    pos[col, 0] = np.resize(tiny, col.sum())
    return pos, a, b


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("case", ["tiny", "negative_zero", "coincident", "huge_rest", "far",
                                  "minus_zero_bound"])
def test_operands_out_of_the_fused_range(gpu, case, resident, collide):
    bodies = [_grid(17, 9), _grid(32, 32, (10.0, 10.0))]
    kw = {}
    if case == "tiny":
        bodies.append(_near_zero(_grid(6, 20, (0.0, -30.0), 0.0)))
    elif case == "negative_zero":
        pos, a, b = _grid(6, 6, (0.0, 0.0), 0.0)
        pos[0] = (-0.0, -0.0)
        bodies.append((pos, a, b))
    elif case == "coincident":
        pos, a, b = _grid(8, 5, (30.0, -40.0))
        pos[9] = pos[8]
        bodies.append((pos, a, b))
    elif case == "huge_rest":
        kw["rest"] = np.float32(3e38)
    elif case == "far":
        pos, a, b = _grid(5, 5)
        pos[3] = (3e19, -2e19)
        bodies.append((pos, a, b))
    sc = _scene(bodies, collide, **kw)
    if case == "minus_zero_bound":
        sc.bounds = (-0.0, -0.0, 60.0, 60.0)
    _check(sc, case, tuning={"resident": resident})


@pytest.mark.parametrize("collide", [0, 1])
def test_equilateral_lattice(gpu, collide):
    """Links of length 1 at 0 and 60 degrees: differences of exactly 0.5 and
    distances of 1 - 2^-24, the significands where a quotient corrected with
    a reciprocal one ulp low comes out wrong."""
    n = 16
    y, x = (v.ravel() for v in np.mgrid[0:n, 0:n])
    pos = np.stack([x + 0.5 * y, y * np.float32(0.8660254)], 1).astype(np.float32)
    a, b = [], []
    for k in range(n * n):
        for dx, dy in ((1, 0), (0, 1), (-1, 1)):
            if 0 <= x[k] + dx < n and y[k] + dy < n:
                a.append(k)
                b.append((y[k] + dy) * n + x[k] + dx)
    sc = _scene([(pos, np.array(a, np.uint64), np.array(b, np.uint64))], collide)
    sc.prev = sc.pos.copy()
    sc.rest[:] = 1.0
    d = pos[a] - pos[b]
    dist = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1])
    assert np.any((dist == np.float32(1.0 - 2.0 ** -24)) & (np.abs(d[:, 0]) == 0.5))
    _check(sc, "equilateral", steps=3)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("stiff", [None, 0.7])
@pytest.mark.parametrize("tuning", [{}, {"t_max": 32}, {"t_max": 96}, {"t_min": 512},
                                    {"resident": 0, "t_max": 64}, {"width_per_thread": 8.0}])
def test_round_widths(gpu, tuning, stiff, mode):
    """Levels of 1 to ~500 ops in rounds of 32 to 512 threads, whole-update
    (bounds + integrate in the same rounds) and link-pass schedules, unit and
    other stiffness, reference and colour order."""
    bodies = [_grid(2, 1, (50.0, 50.0)), _grid(3, 2, (60.0, 50.0)), _grid(33, 31), _grid(32, 3, (-60.0, 40.0)),
              _grid(7, 40, (40.0, -60.0))]
    for collide in (0, 1):
        sc = _scene(bodies, collide, stiff=stiff)
        sc.mode = mode
        _check(sc, f"rounds {tuning} collide {collide}", steps=1, tuning=dict(tuning, serial_width=0.0))


def test_more_bodies_than_multiprocessors(gpu):
    """400 small bodies of two sizes, not packed together: several groups per
    CTA and per multiprocessor, warps without an op skip their round."""
    bodies = [_grid(5 + 3 * (k % 2), 6, (-90.0 + 9.0 * (k % 20), -90.0 + 9.0 * (k // 20)), seed=k)
              for k in range(400)]
    for collide in (0, 1):
        _check(_scene(bodies, collide), f"400 bodies, collide {collide}", steps=2,
               tuning={"pack_np": 1})


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("w,h,mode", [(36, 30, 1), (41, 27, 1), (44, 26, 1), (45, 33, 0), (52, 42, 1)])
def test_levels_a_little_wider_than_the_threads(gpu, w, h, mode, collide):
    """Levels of several rounds, with and without fewer threads for them."""
    sc = _scene([_grid(w, h)], collide, sub_steps=2, link_iters=4, stiff=0.9)
    sc.mode = mode
    _check(sc, f"{w}x{h} mode {mode}", steps=1)

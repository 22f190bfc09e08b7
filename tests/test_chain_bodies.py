"""Chain-like bodies against the oracle: ropes whose passes run behind one
another (by levels), rings replayed in two chains by one thread, and chains
that run in one; every split, lag and mark the planner can choose, and operands
outside the fused solve's range."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state


def _links(pairs):
    a, b = np.array([p[0] for p in pairs]), np.array([p[1] for p in pairs])
    return np.minimum(a, b).astype(np.uint64), np.maximum(a, b).astype(np.uint64)


def _body(kind, n, rng):
    pos = np.stack([np.arange(n) * 0.5, rng.uniform(0.0, 2.0, n)], 1)
    chain = [(i, i + 1) for i in range(n - 1)]
    if kind == "rope":
        pairs = chain
    elif kind == "doubled":
        pairs = chain + chain
    elif kind == "braced":  # a chain, then braces over two particles
        pairs = chain + [(i, i + 2) for i in range(n - 2)]
    elif kind == "hub_last":
        pairs = [(i, (i + 1) % (n - 1)) for i in range(n - 1)] + [(i, n - 1) for i in range(n - 1)]
    else:  # hub first
        pairs = [(1 + i, 1 + (i + 1) % (n - 1)) for i in range(n - 1)] + \
            [(0, 1 + i) for i in range(n - 1)]
    return (pos.astype(np.float32), *_links(pairs))


def _scene(bodies, sub_steps, link_iters, collide=0, stiff=0.8):
    from bendy2d_gb300 import scenes
    placed = [(p + np.float32([3.0, 5.0 + 4.0 * k]), a, b) for k, (p, a, b) in enumerate(bodies)]
    sc = scenes._assemble("chains", placed, bounds=(0.0, 0.0, 400.0, 400.0),
                          sub_steps=sub_steps, link_iters=link_iters, collide=collide)
    sc.stiff = np.full(len(sc.la), stiff, np.float32)
    rng = np.random.default_rng(1)
    sc.prev = scenes._velocity_prev(sc.pos, rng, 0.5, sc.dt / sub_steps)
    return sc


def _check(sc, what, steps=2, tuning=None):
    from oracle import load_scene
    s, o = sc.to_solver(), load_scene(sc)
    if tuning:
        s.set_tuning(**tuning)
    for _ in range(steps):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), what)
    s.close()


def test_plan_ropes_by_levels_and_rings_serially(native_lib):
    rng = np.random.default_rng(2)
    rope = _scene([_body("rope", 200, rng)], 8, 4)
    st = rope.to_solver().plan_stats()
    assert st["serial_bodies"] == 0 and st["ops"] == 8 * (4 * 199 + 200)
    assert st["levels"] < 300
    # too few passes to be wide
    assert _scene([_body("rope", 200, rng)], 1, 1).to_solver().plan_stats()["serial_bodies"] == 1
    for sub in (1, 8, 20):
        for it in (1, 2, 8):
            for kind in ("hub_last", "hub_first"):
                st = _scene([_body(kind, 120, rng)], sub, it).to_solver().plan_stats()
                assert st["serial_bodies"] == 1, (kind, sub, it)


@pytest.mark.gpu
@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("sub_steps,link_iters", [(1, 1), (1, 3), (3, 1), (4, 2)])
@pytest.mark.parametrize("tuning", [{}, {"serial_width": 1e9}, {"serial_width": 0.0},
                                    {"serial_width": 1e9, "stage_frac": 0.0}])
def test_chains_match_oracle(gpu, tuning, sub_steps, link_iters, collide):
    rng = np.random.default_rng(3)
    sizes = [3, 4, 17, 18, 35, 64, 150]
    bodies = [_body(k, n, rng) for k in ("rope", "doubled", "braced", "hub_last", "hub_first")
              for n in sizes]
    sc = _scene(bodies, sub_steps, link_iters, collide)
    _check(sc, f"chains {tuning} {sub_steps}x{link_iters} collide {collide}", tuning=tuning)


@pytest.mark.gpu
@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("case", ["tiny", "negative_zero", "coincident", "huge_rest"])
def test_serial_operands_out_of_the_fused_range(gpu, case, collide):
    """Bodies of one pack: the one out of range is replayed with the IEEE
    intrinsics, its neighbours keep their results."""
    rng = np.random.default_rng(4)
    bodies = [_body(k, n, rng) for k in ("hub_last", "braced") for n in (20, 41)]
    sc = _scene(bodies, 3, 2, collide)
    k = len(bodies[0][0])
    if case == "tiny":
        sc.pos[k:k + 6, 0] = [0.0, 1e-20, 3e-18, 1e-40, 4e-16, 2e-13]
    elif case == "negative_zero":
        sc.pos[k] = (-0.0, -0.0)
    elif case == "coincident":
        sc.pos[k + 3] = sc.pos[k + 2]
    else:
        sc.rest[len(bodies[0][1]) + 5] = np.float32(2e38)
    _check(sc, case, tuning={"serial_width": 1e9})

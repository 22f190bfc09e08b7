"""Serial bodies whose consecutive links share a particle, which the executor
carries in registers: every way a link can hand one on, either end of a link, in one chain and in two, beside bodies that cannot be carried, staged
and streamed records, operands for the general solve.  Bit-exact against the
oracle."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


def _pairs(kind, n, rng):
    chain = [(i, i + 1) for i in range(n - 1)]
    if kind == "rope":
        return chain
    if kind == "ring":
        return chain + [(0, n - 1)]
    if kind == "star":
        return [(i, n - 1) for i in range(n - 1)]
    if kind == "rim_spokes":
        return [(i, (i + 1) % (n - 1)) for i in range(n - 1)] + [(i, n - 1) for i in range(n - 1)]
    if kind == "spokes_rim":
        return [(0, 1 + i) for i in range(n - 1)] + [(1 + i, 1 + (i + 1) % (n - 1))
                                                     for i in range(n - 1)]
    if kind == "comb":  # each tooth, then on to the next: kept, handed on, kept ...
        spine = list(range(0, n, 2))
        out = []
        for i, p in enumerate(spine):
            if p + 1 < n:
                out.append((p, p + 1))
            if i + 1 < len(spine):
                out.append((p, spine[i + 1]))
        return out
    if kind == "doubled":  # the same pair twice in a row: cannot be carried
        return [p for p in chain for _ in range(2)]
    return [(rng.integers(0, i), i) for i in rng.permutation(np.arange(1, n))]  # a tree, any order


def _scene(kinds, turn, sub_steps=3, link_iters=2, collide=0, neg0=False):
    from bendy2d_gb300 import scenes
    rng = np.random.default_rng(7)
    bodies = []
    for k, (kind, n) in enumerate(kinds):
        p = np.array(_pairs(kind, n, rng), np.int64).reshape(-1, 2)
        if turn:  # the particles numbered backwards or at random
            p = (np.arange(n)[::-1] if turn == 2 else rng.permutation(n))[p]
        p = np.sort(p, axis=1)
        pos = np.stack([np.arange(n) * 0.4, rng.uniform(0.0, 2.0, n)], 1) + [4.0, 5.0 + 4.0 * k]
        bodies.append((pos, p[:, 0].astype(np.uint64), p[:, 1].astype(np.uint64)))
    sc = scenes._assemble("carried", bodies, bounds=(0.0, 0.0, 300.0, 300.0), sub_steps=sub_steps,
                          link_iters=link_iters, collide=collide)
    sc.stiff = np.where(np.arange(len(sc.la)) % 2 == 0, np.float32(0.7), np.float32(1.0))
    if neg0:
        sc.pos[0, 0] = -0.0
    sc.prev = scenes._velocity_prev(sc.pos, np.random.default_rng(1), 0.5, sc.dt / sub_steps)
    return sc


def _check(scs, what, **tuning):
    from bendy2d_gb300 import Batch
    from oracle import load_scene
    solvers, oracles = [sc.to_solver() for sc in scs], [load_scene(sc) for sc in scs]
    batch = Batch(solvers)
    batch.set_tuning(serial_width=1000.0, **tuning)
    for _ in range(2):
        batch.update(scs[0].dt)
        for sc, o in zip(scs, oracles):
            assert o.update(sc.dt) == 0
    for s, o in zip(solvers, oracles):
        assert_same_state(solver_state(s), oracle_state(o), what)
    batch.close()


KINDS = ["rope", "ring", "star", "rim_spokes", "spokes_rim", "comb", "doubled", "tree"]


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("turn", [0, 1, 2])
@pytest.mark.parametrize("kind", KINDS)
def test_one_kind_of_many_lengths(gpu, kind, turn, collide):
    lengths = [3, 4, 5, 7, 8, 9, 16, 17, 33, 60, 61, 150]
    _check([_scene([(kind, n)], turn, collide=collide) for n in lengths], f"{kind} turned {turn}")


@pytest.mark.parametrize("stage_frac", [0.0, 2.0])
@pytest.mark.parametrize("sub_steps,link_iters", [(1, 1), (1, 5), (4, 1)])
def test_kinds_side_by_side(gpu, sub_steps, link_iters, stage_frac):
    mixed = [(k, 20 + 7 * i) for i, k in enumerate(KINDS)]
    carried = [(k, 30 + 5 * i) for i, k in enumerate(KINDS[:6])]
    _check([_scene(mixed, 1, sub_steps, link_iters), _scene(carried, 1, sub_steps, link_iters),
            _scene(carried[::-1], 2, sub_steps, link_iters)], "side by side",
           stage_frac=stage_frac)


@pytest.mark.parametrize("kind", KINDS[:6])
def test_a_coordinate_minus_zero(gpu, kind):
    _check([_scene([(kind, 40)], 1, neg0=True), _scene([(kind, 41)], 1)], f"{kind} with -0")

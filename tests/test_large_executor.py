"""The large-body executor: one CTA, clusters, whole updates and link passes,
16-bit and wide ops; the bodies that the flow executor does not take.
Bit-exact against the oracle, on the executor that the case names."""
import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

pytestmark = pytest.mark.gpu


def _cloth(w, h, scatter):
    from bendy2d_gb300 import scenes
    pos, a, b = scenes.grid_body(w, h, (5.0, 5.0), 1.0, 0.01, np.random.default_rng(w))
    if scatter:  # numbered at random: every CTA's particles reach over the whole body
        to = np.random.default_rng(9).permutation(len(pos))
        out = np.empty_like(pos)
        out[to] = pos
        x, y = to[a.astype(np.int64)], to[b.astype(np.int64)]
        pos, a, b = out, np.minimum(x, y).astype(np.uint64), np.maximum(x, y).astype(np.uint64)
    return pos, a, b


def _executors(s, dt):
    """The executors that one update launches, and that update done."""
    s.set_profiling(True)
    s.update(dt)
    names = {k for k in s.profile() if k.startswith("exec_")}
    s.set_profiling(False)
    return names


def _check(sc, executor, tuning):
    from oracle import load_scene
    s, o = sc.to_solver(), load_scene(sc)
    s.set_tuning(**tuning)
    assert _executors(s, sc.dt) == {executor}
    assert o.update(sc.dt) == 0
    s.update(sc.dt)
    assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), f"{executor} {tuning}")
    s.close()


def _scene(w, h, scatter, collide, stiff=None, sub_steps=2, link_iters=2, mode=0):
    from bendy2d_gb300 import scenes
    sc = scenes._assemble("large", [_cloth(w, h, scatter)], bounds=(0.0, 0.0, 300.0, 300.0),
                          sub_steps=sub_steps, link_iters=link_iters, collide=collide)
    sc.prev = scenes._velocity_prev(sc.pos, np.random.default_rng(2), 0.5, sc.dt / sub_steps)
    if stiff is not None:
        sc.stiff = np.full(len(sc.la), stiff, np.float32)
    return sc


@pytest.mark.parametrize("collide", [0, 1])
@pytest.mark.parametrize("w,h,stiff", [(2, 2, None), (9, 7, 0.7), (40, 33, None), (72, 72, 0.7),
                                       (90, 91, None)])
def test_one_cta(gpu, w, h, stiff, collide):
    sc = _scene(w, h, False, collide, stiff, sub_steps=3, link_iters=3)
    _check(sc, f"exec_large_{'links' if collide else 'full'}",
           {"smem_max": 0, "large_max": 1, "serial_width": 0.0})


@pytest.mark.parametrize("w,h,scatter,collide,tuning", [
    (250, 250, False, 0, {}),             # whole update: more than eight CTAs of the flow executor
    (140, 140, True, 0, {}), (141, 139, True, 0, {}),  # whole update: three CTAs
    (200, 200, True, 1, {}),              # link passes: three CTAs
    (260, 260, False, 0, {"large_max": 16}),  # whole update with wide ops: nine CTAs
    (260, 256, True, 1, {}),              # link passes with wide ops: five CTAs
])
def test_clusters(gpu, w, h, scatter, collide, tuning):
    _check(_scene(w, h, scatter, collide), f"exec_large_{'links' if collide else 'full'}", tuning)


@pytest.mark.parametrize("collide", [0, 1])
def test_bodies_of_the_flow_executor_do_not_come_here(gpu, collide):
    _check(_scene(100, 100, False, collide), f"exec_flow_{'links' if collide else 'full'}", {})

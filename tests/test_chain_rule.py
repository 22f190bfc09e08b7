"""Which executor a long chain is planned to, by its length, its passes and its
numbering: serially, or by levels on the executor that holds it."""
import numpy as np
import pytest


def _stats(n, collide, sub_steps, link_iters, scatter=False, tuning=None):
    from bendy2d_gb300 import scenes
    i = np.arange(n)
    pos = np.stack([5.0 + 0.5 * (i % 1000), 5.0 + i // 1000], 1).astype(np.float32)
    at = np.random.default_rng(1).permutation(n) if scatter else i
    out = np.empty_like(pos)
    out[at] = pos
    a, b = at[:-1], at[1:]
    body = (out, np.minimum(a, b).astype(np.uint64), np.maximum(a, b).astype(np.uint64))
    s = scenes._assemble("rope", [body], bounds=(0.0, 0.0, 600.0, 600.0), sub_steps=sub_steps,
                         link_iters=link_iters, collide=collide).to_solver()
    if tuning:
        s.set_tuning(**tuning)
    st = s.plan_stats()
    s.close()
    return {k: st[f"{k}_bodies"] for k in ("serial", "large", "global") if st[f"{k}_bodies"]}


@pytest.mark.parametrize("case,expect", [
    # n, collide, sub_steps, link_iters: the rope is link_iters wide in a link pass
    ((200, 1, 1, 4), {}),                     # one CTA
    ((30000, 1, 1, 2), {"serial": 1}),
    ((30000, 1, 1, 4), {"large": 1}),         # flow executor
    ((70000, 1, 1, 4), {"serial": 1}),        # large-body executor
    ((70000, 1, 1, 6), {"serial": 1}),
    ((70000, 1, 1, 8), {"large": 1}),
    ((140000, 1, 1, 4), {"global": 1}),       # past eight CTAs
    ((70000, 0, 1, 1), {"serial": 1}),
    ((70000, 0, 2, 1), {"global": 1}),
    ((30000, 0, 2, 1, True), {"serial": 1}),  # no CTA of the flow executor holds it
    ((30000, 0, 4, 2, True), {"large": 1}),
    ((30000, 0, 2, 1), {"large": 1}),         # flow executor
    ((30000, 0, 2, 1, True, {"large_max": 0}), {"global": 1}),
    ((70000, 1, 1, 4, False, {"serial_width": 0.0}), {"large": 1}),
    ((70000, 1, 1, 8, False, {"serial_width": 1e9}), {"serial": 1}),
])
def test_chain_executors(native_lib, case, expect):
    assert _stats(*case) == expect

"""Circle and polygon worlds around the sizes where their staged copy meets
the shared memory requested for it: 32 bytes per circle (position, previous
position, acceleration, radius, static flag), and the 16-byte rounding of every
array.  Bit-exact against the oracle."""
import re
from pathlib import Path

import numpy as np
import pytest

from helpers import assert_same_state, oracle_state, solver_state

CSRC = Path(__file__).resolve().parents[1] / "bendy2d_gb300" / "csrc"


def _staged_bytes(nc, ncl, polys):
    """The arrays that stage_view lays out, each rounded to 16 bytes."""
    ng, nv = len(polys), sum(polys)
    nst = ng * (ng - 1) + 1 if ng >= 2 else 0
    parts = [16 * ng, 24 * ng, 8 * ng, 8 * nc, 8 * nc, 8 * nc, 8 * nv, 8 * nv, 8 * nv, 8 * ncl,
             8 * nv, 4 * nc, 4 * nc, 4 * ncl, 4 * nv, 4 * nst, 4 * nst]
    return sum((p + 15) & ~15 for p in parts)


def test_requested_shared_memory_covers_the_staged_arrays():
    """Both expressions of the request, read from the sources, are at least
    what the layout takes, for every circle count up to 400."""
    dev = re.search(r"return (48u \* v\.ng[^;]*);", (CSRC / "kernels.cuh").read_text()).group(1)
    host = re.search(r"need = (48 \* ng[^;]*);", (CSRC / "engine.cu").read_text()).group(1)
    dev = re.sub(r"(\d+)u", r"\1", " ".join(dev.split())).replace("v.", "")
    host = (" ".join(host.split()).replace("im.clab.size()", "ncl").replace("im.plab.size()", "npl")
            .replace("im.stage_off.size()", "nst"))
    for nc in range(0, 400):
        for ng in (0, 1, 2, 7, 33):
            polys = [3 + k % 6 for k in range(ng)]
            env = dict(nc=nc, ng=ng, ncl=nc // 2, nv=sum(polys), npl=sum(polys),
                       nst=ng * (ng - 1) + 1 if ng >= 2 else 0)
            need = _staged_bytes(nc, nc // 2, polys)
            assert eval(dev, {}, env) >= need and eval(host, {}, env) >= need, (nc, ng)


@pytest.mark.gpu
@pytest.mark.parametrize("n_circles,n_polys", [(49, 0), (64, 32), (101, 2), (200, 5)])
def test_worlds_with_many_circles_match_oracle(gpu, n_circles, n_polys):
    from bendy2d_gb300 import scenes
    from oracle import load_scene
    rng = np.random.default_rng(n_circles)
    box = 30.0 * np.sqrt(n_circles)
    polys = [{"points": scenes.convex_polygon(rng, rng.uniform(20, box - 20, 2),
                                              rng.uniform(5, 15), 4 + k % 5), "static": False}
             for k in range(n_polys)]
    circles = [scenes._circle(rng.uniform(0, box, 2), rng.uniform(2, 9), k % 5 == 0)
               for k in range(n_circles)]
    sc = scenes._assemble("many", [], circles=circles, polygons=polys, bounds=(0.0, 0.0, box, box),
                          sub_steps=3, link_iters=1)
    s, o = sc.to_solver(), load_scene(sc)
    for _ in range(4):
        s.update(sc.dt)
        assert o.update(sc.dt) == 0
    assert_same_state(solver_state(s), oracle_state(o), f"{n_circles} circles")
    s.close()

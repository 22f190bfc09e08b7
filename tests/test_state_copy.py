"""The state to and from host memory: page-locked and pageable, aligned and
not, byte counts that are and are not multiples of 16, one world and several
in an engine.  Every route moves the same bytes, in the stream's order."""
import numpy as np
import pytest

from helpers import solver_state

pytestmark = pytest.mark.gpu


def _solver(n, circles):
    from bendy2d_gb300 import scenes
    pos, a, b = scenes.grid_body(n, 3, (5.0, 5.0), 1.0, 0.01, np.random.default_rng(n))
    return scenes._assemble("state", [(pos, a, b)], bounds=(0.0, 0.0, 400.0, 60.0), sub_steps=2,
                            link_iters=2,
                            circles=[scenes._circle((9.0 + 7 * k, 40.0), 2.0, False)
                                     for k in range(circles)]).to_solver()


def _buffers(n, kind):
    """A buffer of n bytes as (owner, uint8 view, address)."""
    import torch
    off = 4 if kind == "unaligned" else 0
    t = torch.zeros(n + 64, dtype=torch.uint8, pin_memory=kind != "pageable")
    v = t.numpy()
    off += -v.ctypes.data % 16
    return t, v[off:off + n], v.ctypes.data + off


@pytest.mark.parametrize("kind", ["pinned", "pageable", "unaligned"])
@pytest.mark.parametrize("n,circles,many", [(2, 0, False), (7, 1, False), (64, 2, False),
                                            (300, 5, False), (7, 1, True)])
def test_every_route_moves_the_same_bytes(gpu, n, circles, many, kind):
    import torch
    from bendy2d_gb300 import Batch
    solvers = [_solver(n + k, circles) for k in range(3 if many else 1)]
    batch = Batch(solvers) if many else None
    stream = torch.cuda.Stream()
    (batch or solvers[0]).set_stream(stream.cuda_stream)
    update = (batch or solvers[0]).update
    sizes = [s.state_bytes() for s in solvers]
    start = [_buffers(k, kind) for k in sizes]
    for s, (_, _, at) in zip(solvers, start):
        s.state_download_async(at)
    runs = []
    for _ in range(2):  # the same start twice: the same end
        out = [_buffers(k, kind) for k in sizes]
        for s, (_, _, at) in zip(solvers, start):
            s.state_upload_async(at)
        update(1.0 / 60.0)
        for s, (_, _, at) in zip(solvers, out):
            s.state_download_async(at)
        torch.cuda.synchronize()
        runs.append(out)
    for k, s in enumerate(solvers):
        first, second = runs[0][k][1], runs[1][k][1]
        assert first.tobytes() == second.tobytes() != start[k][1].tobytes()
        pos = np.ascontiguousarray(solver_state(s)[0], np.float32)
        assert first[:pos.nbytes].tobytes() == pos.tobytes()

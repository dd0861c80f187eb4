"""The drivers of a small hierarchy's first solve with use_graph = 1: it starts on the stream, and when its
first iterations say that many are left the rest runs as a graph of the loop. The iterates are those of the
stream driver (use_graph = 0) and of the captured solve (the second solve), bit for bit; the kernels launched
tell the drivers apart: the graph's loop has a kernel that sets its condition, the stream enqueues one
iteration past the last."""
import numpy as np
import pytest

from test_gpu_parity import fcg
from test_gpu_stencil import diffusion

pytestmark = pytest.mark.gpu


def solves(bx, A, b, k, **kw):
    """k solves with one hierarchy: solution, info and kernels launched of each."""
    h = bx.prec_setup(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, fcg(bx, **kw))
    out = []
    for _ in range(k):
        c0 = bx.lib().bcmgx_launch_count()
        x, info = h.solve(b)
        out.append((x, info, bx.lib().bcmgx_launch_count() - c0))
    h.free()
    return out


# many iterations (the loop's graph); the same cut off by itnlim at an odd and an even number; few (no graph)
@pytest.mark.parametrize("kw,graph", [(dict(rtol=1e-12), True), (dict(rtol=1e-12, itnlim=17), True),
                                      (dict(rtol=1e-12, itnlim=18), True), (dict(rtol=1e-3), False)])
@pytest.mark.parametrize("prec", ["FP64", "FP32"])
def test_first_solve(bx, cuda, kw, graph, prec):
    A = diffusion(bx, (24, 22, 26))
    b = A @ np.random.default_rng(5).uniform(-1, 1, A.shape[0])
    (x0, i0, l0), = solves(bx, A, b, 1, use_graph=0, vcycle_precision=prec, **kw)
    (x1, i1, l1), (x2, i2, l2) = solves(bx, A, b, 2, use_graph=1, vcycle_precision=prec, **kw)
    assert i0["niter"] == i1["niter"] == i2["niter"] and i0["status"] == i1["status"] == i2["status"]
    assert np.array_equal(x0, x1) and np.array_equal(x0, x2)
    assert i0["exit_res"] == i1["exit_res"] == i2["exit_res"]
    if graph:
        assert i0["niter"] > 16
        assert l1 != l0   # not the stream driver's kernels to the end
    else:
        assert l1 == l0
    assert l2 != l0 or i0["niter"] % 2 == 0


def test_breakdown_in_a_later_solve(bx, cuda):
    """A NaN in the right-hand side of the first solve (the stream), and of one that the captured graph runs."""
    A = diffusion(bx, (14, 13, 12))
    n = A.shape[0]
    h = bx.prec_setup(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, fcg(bx, rtol=1e-8))
    xs = np.random.default_rng(0).uniform(-1, 1, n)
    bad = np.ones(n)
    bad[n // 3] = np.nan
    for _ in range(3):
        with pytest.raises(bx.BcmgxError) as e:
            h.solve(bad)
        assert e.value.code == -7   # BCMGX_ERR_NOT_SPD
        x, info = h.solve(A @ xs)
        assert info["status"] == 0 and np.linalg.norm(x - xs) < 1e-5 * np.linalg.norm(xs)
    h.free()

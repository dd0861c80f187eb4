"""The candidate ranks of the set-up's matching (k_rank_rows with the weights formed in registers) order a row by the
arguments of the logarithms and fall back to the logarithms where two arguments are within 1e-12 of each other:
there different arguments may have one logarithm, and the column decides. Compared with the matching on the stored
weights (bcmgx_edge_weights, the logarithms themselves)."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_parity import fcg

pytestmark = pytest.mark.gpu


def near_ties(offs, n, ulps, seed):
    """A band of couplings around -1 that differ by up to `ulps` units in the last place, and a diagonal of 0.002: the
    arguments 1 + 2 |a| / 0.004 are near 501, a coupling's step moves one by 1.1e-13 and its logarithm by a quarter of the
    logarithm's last place, 8.9e-16. (Only matched, not solved.)"""
    rng = np.random.default_rng(seed)
    B = sp.diags([-(1.0 + 2.0 ** -52 * rng.integers(0, ulps, n - o)) for o in offs], offs)
    A = (B + B.T + sp.diags(np.full(n, 0.002))).tocsr()
    A.sort_indices()
    return A


# rows of at most 8, 16 and 32 entries (a sub-warp of lanes each), one row past the last warp's, and a single warp
@pytest.mark.parametrize("offs", [(1, 40, 200), (1, 2, 3, 40, 41, 200), tuple(range(1, 14))])
@pytest.mark.parametrize("n,ulps", [(4097, 9), (4097, 400), (300, 9)])
def test_near_ties_by_logarithm(bx, oracle, cuda, offs, n, ulps):
    import torch
    A = near_ties(offs, n, ulps, 3)
    row, col, val = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    d = [torch.from_numpy(a).to(cuda) for a in (row, col, val)]
    W, _ = bx.edge_weights(*d, torch.ones(n, dtype=torch.float64, device=cuda))
    want = bx.suitor_matching(d[0], d[1], W).cpu().numpy()
    # the case is there: the order by the arguments gives another matching
    args = 1.0 - 2.0 * val / 0.004
    mo = oracle.Matrix.from_csr(A.indptr, A.indices, A.data)
    assert not np.array_equal(mo.match(args, 0), want) and np.array_equal(mo.match(W.cpu().numpy(), 0), want)
    h = bx.prec_setup(row, col, val, fcg(bx, record_sweeps=1, max_levels=2, aggrsweeps=0))
    got = h.sweeps()[0]["match"]
    h.free()
    assert np.array_equal(got, want)

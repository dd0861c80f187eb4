"""The stencil row kernels (stencil.cuh: columns from one list of offsets, one form byte per row) against
the plain row kernel with one thread per row (rowops.cuh k_rowop<1>). Both add each row's entries in CSR
order with the same multiply-adds, so whole set-ups and solves must agree bit for bit. BCMGX_TPR=65 forces
the stencil kernels on every level that has the form (the sliced ones on the others), BCMGX_TPR=1 the plain
kernel."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_parity import fcg
from test_gpu_staged import matrix, setup_solve

pytestmark = pytest.mark.gpu

STENCIL = 65   # forced; hierarchies report 64, as for the sliced kernels, and index_bytes -1
SLICED = 64


@pytest.fixture(autouse=True)
def multi_launch_cycle(monkeypatch):
    """These tests exercise the cycle's own kernels: the persistent coarse cycle stays off."""
    monkeypatch.setenv("BCMGX_PERSIST_NNZ", "0")


def diffusion(bx, grid):
    k = np.exp(np.random.default_rng(11).standard_normal(grid[0] * grid[1] * grid[2]))
    row, col, val = bx.diffusion_7p(*grid, k)
    return sp.csr_matrix((val, col, row), shape=(row.size - 1,) * 2)


def banded(n, offs, seed):
    """A symmetric diagonally dominant matrix with the given upper offsets, constant along each diagonal for
    seed None, else with values of its own everywhere."""
    rng = np.random.default_rng(seed)
    B = sp.diags([-np.ones(n - o) if seed is None else -rng.uniform(0.5, 1.5, n - o) for o in offs], offs)
    B = B + B.T
    d = np.full(n, 2.0 * len(offs) + 1.0) if seed is None else np.asarray(-B.sum(axis=1)).ravel() + 1.0
    return (B + sp.diags(d)).tocsr()


# (matrix, does level 0 have the form): table and stored values; 7 and 27 offsets and symmetric bands of 3, 9, 15, 17,
# 29 and 31, the least and most odd counts of the compiled widths (8, 16, 28 and 32 offsets: a symmetric matrix with a
# diagonal has an odd number); sizes that leave a ragged last slice and block; a matrix smaller than one slice; a matrix
# without the form
CASES = {
    "lap27": (lambda bx: matrix(bx, ("lap27", (37, 29, 23))), True),
    "lap7": (lambda bx: matrix(bx, ("lap7", (33, 31, 25))), True),
    "lap7_small": (lambda bx: matrix(bx, ("lap7", (5, 3, 2))), True),
    "diffusion": (lambda bx: diffusion(bx, (31, 27, 22)), True),
    "band9": (lambda bx: banded(3001, (1, 2, 40, 200), None), True),
    "band9_stored": (lambda bx: banded(4003, (1, 2, 40, 200), 4), True),
    "band3_stored": (lambda bx: banded(999, (1,), 5), True),
    "band15": (lambda bx: banded(3100, (1, 2, 3, 5, 7, 11, 13), None), True),
    "band17": (lambda bx: banded(2050, (1, 2, 3, 5, 7, 11, 13, 17), None), True),
    "band29_stored": (lambda bx: banded(9000, tuple(range(1, 15)), 6), True),
    "band31": (lambda bx: banded(2500, tuple(range(1, 16)), None), True),
    "band33": (lambda bx: banded(2500, tuple(range(1, 17)), None), False),
}


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("name", list(CASES))
def test_stencil_solve_bit_identical(bx, cuda, monkeypatch, name, prec):
    make, has = CASES[name]
    A = make(bx)
    A.sort_indices()
    n = A.shape[0]
    b = A @ np.random.default_rng(3).uniform(-1, 1, n)
    kw = dict(vcycle_precision=prec, rtol=1e-8)
    x0, i0, h0 = setup_solve(bx, monkeypatch, A, b, 1, **kw)
    x1, i1, h1 = setup_solve(bx, monkeypatch, A, b, STENCIL, **kw)
    assert set(h1["tpr"]) == {SLICED} and (h1["index_bytes"][0] == -1) == has
    assert i0["status"] == 0 and i1["status"] == 0
    assert i0["niter"] == i1["niter"]
    assert np.array_equal(x0, x1)


def solve_both(bx, monkeypatch, A, kw):
    b = A @ np.random.default_rng(3).uniform(-1, 1, A.shape[0])
    x0, i0, _ = setup_solve(bx, monkeypatch, A, b, 1, **kw)
    x1, i1, h1 = setup_solve(bx, monkeypatch, A, b, STENCIL, **kw)
    assert h1["index_bytes"][0] == -1
    assert i0["niter"] == i1["niter"] and np.array_equal(x0, x1)


# the box kernel with every number of rows a lane: lines whose number is not a multiple of 2 or of 4 (the last group
# passes the end), lines shorter and longer than a warp, planes of one line less than a group, and a single group
@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("rows", [1, 2, 4])
@pytest.mark.parametrize("grid", [(37, 29, 23), (31, 6, 11), (70, 3, 7), (3, 5, 41), (33, 4, 4)])
def test_box_rows_bit_identical(bx, cuda, monkeypatch, grid, rows, prec):
    monkeypatch.setenv("BCMGX_BOX_ROWS", str(rows))
    solve_both(bx, monkeypatch, matrix(bx, ("lap27", grid)), dict(vcycle_precision=prec, rtol=1e-8))


# the sizes where the rule takes other rows: two and four for the FP32 and FP64 sweeps (64x61x67: 2 and 4, 73x75x72: 4 and
# 2), and two for the product above 3 M rows
@pytest.mark.parametrize("grid,prec", [((64, 61, 67), "FP32"), ((64, 61, 67), "FP64"), ((73, 75, 72), "FP32"),
                                       ((73, 75, 72), "FP64"), ((163, 151, 123), "FP32")])
def test_box_rule_bit_identical(bx, cuda, monkeypatch, grid, prec):
    solve_both(bx, monkeypatch, matrix(bx, ("lap27", grid)), dict(vcycle_precision=prec, rtol=1e-6))


@pytest.mark.parametrize("rows", [0, 2, 4])
def test_stencil_reads_only_a_rows_own_entries(bx, cuda, monkeypatch, rows):
    """One sweep of the preconditioner on a vector with an Inf: the rows that have no entry in its column keep the
    plain kernel's bits (an offset that a row lacks must not bring Inf * 0 into its sum). rows: a lane's in the box
    kernel; 0: the general stencil kernel, which takes a box of this size."""
    import torch
    A = matrix(bx, ("lap27", (21, 19, 17)))
    n = A.shape[0]
    r = np.random.default_rng(5).uniform(-1, 1, n)
    r[n // 2 + 3] = np.inf
    r[20] = np.nan      # the end of an x line: row 21 starts the next one and has no entry there
    t = torch.from_numpy(r).to(cuda)
    monkeypatch.setenv("BCMGX_BOX_ROWS", str(rows))
    outs = []
    for code in (1, STENCIL):
        monkeypatch.setenv("BCMGX_TPR", str(code))
        h = bx.prec_setup(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data,
                          fcg(bx, preconditioner="L1_JACOBI", l1jacsweeps=2))
        monkeypatch.delenv("BCMGX_TPR")
        outs.append(h.prec_apply(t).cpu().numpy())
        h.free()
    assert np.isfinite(outs[0]).sum() > n // 2
    assert np.array_equal(outs[0], outs[1], equal_nan=True)


def test_stencil_code_on_another_matrix(bx, cuda, monkeypatch):
    """The code of a tuned size applied to a matrix of that size without the form: the sliced kernels take it."""
    n = 4000
    rng = np.random.default_rng(8)
    P = sp.random(n, n, 4.0 / n, random_state=np.random.RandomState(2))
    P = -(P + P.T)
    A = (P + sp.diags(np.asarray(-P.sum(axis=1)).ravel() + 1.0)).tocsr()
    A.sort_indices()
    b = A @ rng.uniform(-1, 1, n)
    x0, i0, _ = setup_solve(bx, monkeypatch, A, b, 1, rtol=1e-8)
    x1, i1, h1 = setup_solve(bx, monkeypatch, A, b, STENCIL, rtol=1e-8)
    assert h1["index_bytes"][0] >= 0 and i0["niter"] == i1["niter"] and np.array_equal(x0, x1)


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("grid,k", [((40, 37, 33), 32), ((41, 35, 39), 19), ((70, 61, 66), 4), ((71, 67, 59), 3), ((113, 101, 97), 1)])
def test_stencil_block_solve(bx, cuda, monkeypatch, grid, k, prec):
    """Block solves on a 27-point box (blk_box_rows: two or four rows of a slot share their gathers), with ragged lines,
    planes that are not a multiple of four lines and 1 to 32 columns, against the CSR block kernels. The sweeps
    add the same terms in the same order; the dot products' partial sums do not, so the solutions agree to
    the rounding of those sums (1e-16 each, carried through some 30 iterations)."""
    A = matrix(bx, ("lap27", grid))
    n = A.shape[0]
    B = A @ np.random.default_rng(3).uniform(-1, 1, (n, k))
    out = []
    for code in (1, STENCIL):
        monkeypatch.setenv("BCMGX_TPR", str(code))
        h = bx.prec_setup(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data,
                          fcg(bx, vcycle_precision=prec, rtol=1e-8))
        monkeypatch.delenv("BCMGX_TPR")
        assert (h.info()["index_bytes"][0] == -1) == (code == STENCIL)
        out.append(h.solve_multi(B))
        h.free()
    (X0, i0), (X1, i1) = out
    assert [i["niter"] for i in i0] == [i["niter"] for i in i1]
    assert np.linalg.norm(X1 - X0) <= 1e-11 * np.linalg.norm(X0)
    assert np.linalg.norm(B - A @ X1) <= 1.0001e-8 * np.linalg.norm(B)

"""The input checks (k_validate: 256 rows a block through shared memory, long rows by warps) refuse every
kind of malformed CSR wherever it sits, before anything reads x, and accept what is well formed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tridiagonal(n, dense_rows=()):
    """Row offsets, columns and values of a diagonally dominant matrix; dense_rows have every column."""
    cols = [np.arange(n) if r in dense_rows else np.arange(max(r - 1, 0), min(r + 2, n)) for r in range(n)]
    row = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(row))
    return row, col, np.where(rows == col, 2.0 * n, -1.0)


def spoil(kind, row, col, n, r):
    """The matrix with one fault of `kind` in row r."""
    row, col = row.copy(), col.copy()
    b, e = row[r], row[r + 1]
    if kind == "first offset":
        row[0] = 1
    elif kind == "last offset":
        row[n] -= 1
    elif kind == "decreasing offsets":
        row[r + 1] = row[r] - 1 if r else -1
    elif kind == "offset past the end":
        row[r + 1] = col.size + 7
    elif kind == "negative column":
        col[b] = -1
    elif kind == "column too large":
        col[e - 1] = n
    elif kind == "not ascending":
        col[b] = col[b + 1]
    elif kind == "no diagonal":
        k = b + int(np.searchsorted(col[b:e], r))
        col[k] = col[k - 1] if k > b else col[k + 1]
    return row, col


# 255, 256, 257: a block's rows; 8192 entries: what a block stages (3 * 256 + rows of 3000 columns pass it); 500 rows
# of 500: longer than 32 throughout, so fewer rows a block
SIZES = [(1, ()), (255, ()), (256, ()), (257, ()), (3000, (5, 6, 2999)), (3000, ()), (500, range(500)), (9, range(9))]


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("n,dense", SIZES)
def test_accepts(bx, cuda, n, dense, shift):
    """shift: the columns start that many words past a 16-byte boundary."""
    import torch
    row, col, val = tridiagonal(n, dense)
    x = np.random.default_rng(1).uniform(-1, 1, n)
    t = [torch.from_numpy(a).to(cuda) for a in (row, np.concatenate([np.full(shift, -5, np.int32), col]), val, x)]
    t[1] = t[1][shift:]
    y = bx.spmv(*t, torch.empty(n, dtype=torch.float64, device=cuda)).cpu().numpy()
    import scipy.sparse as sp
    want = sp.csr_matrix((val, col, row), shape=(n, n)) @ x
    # FP64 sums of at most n terms in another order
    assert np.abs(y - want).max() <= n * 2.3e-16 * (np.abs(val).max() + n)
    h = bx.prec_setup(row, col, val, bx.params_default(solver="FCG", preconditioner="BCMG", dispnorm=0))
    assert h.info()["n"][0] == n
    h.free()


@pytest.mark.parametrize("kind", ["first offset", "last offset", "decreasing offsets", "offset past the end",
                                  "negative column", "column too large", "not ascending", "no diagonal"])
@pytest.mark.parametrize("n,dense", [(257, ()), (3000, (5, 6, 2999)), (500, range(500))])
def test_refuses(bx, cuda, n, dense, kind):
    import torch
    row, col, val = tridiagonal(n, dense)
    for r in (0, 5, 255, 256, n - 1):
        bad_row, bad_col = spoil(kind, row, col, n, r)
        with pytest.raises(bx.BcmgxError) as e:
            bx.prec_setup(bad_row, bad_col, val, bx.params_default(solver="FCG", preconditioner="BCMG", dispnorm=0))
        assert e.value.code == -1
        if kind == "no diagonal" and np.all(np.diff(bad_col[row[r]:row[r + 1]]) > 0):
            continue   # the product itself needs no diagonal
        y = torch.full((n,), 3.0, dtype=torch.float64, device=cuda)
        t = [torch.from_numpy(a).to(cuda) for a in (bad_row, bad_col, val, np.ones(n))]
        with pytest.raises(bx.BcmgxError) as e:
            bx.spmv(*t, y)
        assert e.value.code == -1
        assert bool((y == 3.0).all())   # refused before the product

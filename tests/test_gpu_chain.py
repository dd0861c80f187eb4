"""Sweep chains of small levels in one thread-block cluster (chain.cu) against one launch per sweep
(BCMGX_CHAIN=0): the same rows, order of additions and update, so cycles and solves agree bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import ROOT
from test_gpu_batch import _systems
from test_gpu_faults import pool_used_bytes
from test_gpu_parity import fcg
from test_gpu_staged import matrix

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def multi_launch_cycle(monkeypatch):
    """These tests exercise the cycle's own kernels: the persistent coarse cycle stays off."""
    monkeypatch.setenv("BCMGX_PERSIST_NNZ", "0")


def cycle_and_solve(bx, monkeypatch, A, chain, S=2, **kw):
    """One cycle and two solves with S threads per row on every level: the first starts on the stream, the second
    is the captured one (use_graph = 1)."""
    import torch
    monkeypatch.setenv("BCMGX_CHAIN", chain)
    monkeypatch.setenv("BCMGX_TPR", str(S))
    n = A.shape[0]
    h = bx.prec_setup(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data,
                      fcg(bx, rtol=1e-8, **kw))
    rng = np.random.default_rng(7)
    r = rng.uniform(-1, 1, n)
    c0 = bx.lib().bcmgx_launch_count()
    v = h.prec_apply(torch.from_numpy(r).cuda()).cpu().numpy()
    launches = bx.lib().bcmgx_launch_count() - c0
    # (one row: the start-up step is exact and leaves a zero residual, which the iteration refuses)
    x, info = v, {"niter": 1}
    if n > 1:
        b = A @ rng.uniform(-1, 1, n)
        x, info = h.solve(b)
        x2, info2 = h.solve(b)
        assert info2["niter"] == info["niter"] and np.array_equal(x, x2)
    h.free()
    return v, x, info, launches


# one row; a block's first rows (1 block), several blocks, the largest cluster; rows of 7 and 27 entries, random
# columns (every block in every other's halo), a dense row, and a level too large for a cluster (it keeps its launches)
CASES = {
    "one_row": lambda bx: sp.identity(1, format="csr") * 3.0,
    "lap7_tiny": lambda bx: matrix(bx, ("lap7", (5, 3, 2))),
    "lap7": lambda bx: matrix(bx, ("lap7", (13, 11, 9))),
    "lap27": lambda bx: matrix(bx, ("lap27", (17, 13, 11))),
    "lap27_16": lambda bx: matrix(bx, ("lap27", (23, 21, 19))),
    "rand": lambda bx: matrix(bx, ("rand", (5000, 0.003, 2, True))),
    "arrow": lambda bx: matrix(bx, ("arrow", (3000, 4, 5))),
    "diff": lambda bx: matrix(bx, ("diff", (24, 3))),
    "lap7_large": lambda bx: matrix(bx, ("lap7", (40, 40, 40))),
}


@pytest.mark.parametrize("prec", ["FP64", "FP32"])
@pytest.mark.parametrize("name,S", [(k, 2) for k in CASES] + [(k, S) for k in ("lap7", "lap27_16", "rand") for S in (1, 4, 8, 16)])
def test_chain_bit_identical(bx, cuda, monkeypatch, name, S, prec):
    A = CASES[name](bx)
    A.sort_indices()
    v0, x0, i0, l0 = cycle_and_solve(bx, monkeypatch, A, "0", S, vcycle_precision=prec)
    v1, x1, i1, l1 = cycle_and_solve(bx, monkeypatch, A, "1", S, vcycle_precision=prec)
    assert np.array_equal(v0, v1)
    assert i0["niter"] == i1["niter"] and np.array_equal(x0, x1)
    if name.startswith("lap"):
        assert l1 < l0   # the coarsest level's chain at least is one launch


@pytest.mark.parametrize("kw", [dict(cycle_type="W_CYCLE"), dict(cycle_type="H_CYCLE"), dict(relaxnumber_coarse=2),
                                dict(prerelax_sweeps=1, postrelax_sweeps=2), dict(prerelax_sweeps=0, postrelax_sweeps=3),
                                dict(use_graph=0)])
def test_chain_cycles(bx, cuda, monkeypatch, kw):
    """Second visits of a level (a chain from its iterate), chains of 1 to 3 sweeps, the stream driver alone."""
    A = matrix(bx, ("lap7", (40, 37, 33)))
    v0, x0, i0, _ = cycle_and_solve(bx, monkeypatch, A, "0", **kw)
    v1, x1, i1, _ = cycle_and_solve(bx, monkeypatch, A, "1", **kw)
    assert np.array_equal(v0, v1) and i0["niter"] == i1["niter"] and np.array_equal(x0, x1)


def test_plan_memory(bx, cuda, monkeypatch):
    """A plan holds its level's entries (10 bytes each, rows padded to a slice's longest and blocks to the widest),
    lists of what blocks exchange and nothing more: at most 64 bytes for an entry of the coarse levels."""
    import torch
    row, col, val = bx.laplacian_3d(7, 24, 24, 24)
    p = fcg(bx, rtol=1e-8, autotune=0)
    held, entries = [], 0
    for chain in ("0", "0", "1"):   # (the first set-up fills the process-wide caches)
        monkeypatch.setenv("BCMGX_CHAIN", chain)
        torch.cuda.synchronize()
        base = pool_used_bytes()
        h = bx.prec_setup(row, col, val, p)
        torch.cuda.synchronize()
        held.append(pool_used_bytes() - base)
        entries = sum(h.info()["nnz"][1:])
        h.free()
    assert 0 < held[2] - held[1] <= 64 * entries


def test_batch_members_have_no_plans(bx, cuda, monkeypatch):
    """A batch's members take no memory for chains that its solves never run, and one handed out to be solved
    alone has them."""
    import torch
    systems = _systems(bx, 12, 4)
    b = torch.from_numpy(np.random.default_rng(5).uniform(-1, 1, systems[3][0].size - 1)).to(cuda)
    held, launches, xs = [], [], []
    for chain in ("0", "0", "1"):
        monkeypatch.setenv("BCMGX_CHAIN", chain)
        torch.cuda.synchronize()
        base = pool_used_bytes()
        B = bx.Batch(systems, fcg(bx, rtol=1e-8), nthreads=4)
        torch.cuda.synchronize()
        held.append(pool_used_bytes() - base)
        c0 = bx.lib().bcmgx_launch_count()
        x, info = B.hierarchy(3).solve(b)
        launches.append(bx.lib().bcmgx_launch_count() - c0)
        xs.append((info["niter"], x.cpu().numpy()))
        B.free()
    assert held[2] == held[1]
    assert launches[2] < launches[1]
    # two threads per row instead of four: sums in another order
    assert xs[2][0] == xs[1][0] and np.linalg.norm(xs[2][1] - xs[1][1]) <= 1e-8 * np.linalg.norm(xs[1][1])


# The CUDA runtime's calls that a context without room for a cluster of more than 8 blocks answers with an error:
# the launch and the occupancy query. Everything else goes to the runtime.
NO_LARGE_CLUSTER = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
static unsigned blocks(const cudaLaunchConfig_t* c)
{
    for (unsigned i = 0; c && i < c->numAttrs; i++)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) return c->attrs[i].val.clusterDim.x;
    return 1;
}
static void* next(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a)
{
    if (blocks(c) > 8) return cudaErrorInvalidConfiguration;
    return ((cudaError_t(*)(const cudaLaunchConfig_t*, const void*, void**))next("cudaLaunchKernelExC"))(c, f, a);
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c)
{
    if (blocks(c) > 8) { *n = 0; return cudaSuccess; }
    return ((cudaError_t(*)(int*, const void*, const cudaLaunchConfig_t*))next("cudaOccupancyMaxActiveClusters"))(n, f, c);
}
"""

CHILD = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import bootcmatchgx_b200 as bx
row, col, val = bx.laplacian_3d(27, 23, 21, 19)
h = bx.prec_setup(row, col, val, bx.params_default(solver="FCG", preconditioner="BCMG", dispnorm=0, rtol=1e-8))
c0 = bx.lib().bcmgx_launch_count()
x, info = h.solve(np.random.default_rng(3).uniform(-1, 1, row.size - 1))
print(info["status"], info["niter"], bx.lib().bcmgx_launch_count() - c0, x.tobytes().hex())
"""


def test_no_large_cluster(cuda, tmp_path):
    """Where no cluster of 16 blocks can run, set-up succeeds and the level keeps one launch per sweep."""
    src, lib = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(NO_LARGE_CLUSTER)
    subprocess.run(["gcc", "-shared", "-fPIC", "-I/usr/local/cuda/include", str(src), "-o", str(lib), "-ldl"], check=True)

    def child(**env):
        e = {k: v for k, v in os.environ.items() if k not in ("BCMGX_CHAIN", "BCMGX_TPR")}
        r = subprocess.run([sys.executable, "-c", CHILD, ROOT], env={**e, **env}, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout.split()

    launches, without, with_chain = child(BCMGX_CHAIN="0"), child(LD_PRELOAD=str(lib)), child()
    assert without == launches and launches[0] == "0"
    assert int(with_chain[2]) < int(launches[2])   # the level has a chain of 16 blocks where it may


@pytest.mark.parametrize("grid,chain", [((40, 40, 40), True), ((44, 44, 44), True), ((48, 48, 48), False)])
def test_chain_stops_where_launches_are_faster(bx, cuda, monkeypatch, grid, chain):
    """Coarsest levels of 8,000, 10,648 and 13,824 rows of 7 entries (two levels): the last has more than two
    slices a warp and 93,312 entries, and keeps one launch per sweep."""
    A = matrix(bx, ("lap7", grid))
    _, x0, _, l0 = cycle_and_solve(bx, monkeypatch, A, "0", max_levels=2)
    _, x1, _, l1 = cycle_and_solve(bx, monkeypatch, A, "1", max_levels=2)
    assert (l1 < l0) == chain and np.array_equal(x0, x1)

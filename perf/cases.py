"""Timed cases of the solver library: the calls that user programs make, over the range of sizes, matrices and options they
make them with. A case is a dict of plain values; its "what" names the call:

  step     prec_setup + solve + prec_finalize of one system (a Newton or time step that changes the matrix)
  solve    one solve with a kept hierarchy (new right-hand side, same matrix)
  multi    one block solve of "k" right-hand sides with a kept hierarchy
  batch    one solve of "m" uneven systems with a kept batch
  grad     autograd: set-up, forward solve, adjoint solve; gradients of the matrix values and of b
  prec     one preconditioner application (a user's own Krylov loop)
  spmv     y = A x on the caller's CSR arrays
  match    edge weights and suitor matching on the caller's CSR arrays

Matrices are boxes of nx * ny * nz cells, x fastest: "poisson7" / "poisson27" (diagonal 6 / 26, off-diagonals -1, Dirichlet)
and "diffusion7" (7-point finite volumes, kappa = exp(theta), theta a Gaussian random field with squared-exponential covariance
of length 8 cells and sigma 2, harmonic-mean faces). Right-hand sides are b = A x* with x* uniform in [-1, 1], so the exact
solution is x*."""
import math

import torch

import bootcmatchgx_b200 as bx
from bootcmatchgx_b200 import autograd

DEV = "cuda"


def listed():
    return [
        # the smallest step: the 10^3 box of the generator's sample files, all latency
        {"name": "poisson7_10_step", "what": "step", "matrix": "poisson7", "nx": 10, "ny": 10, "nz": 10, "cycle": "FP64"},
        # a small system set up and solved once, every level inside L2
        {"name": "poisson7_50_step", "what": "step", "matrix": "poisson7", "nx": 50, "ny": 50, "nz": 50, "cycle": "FP64"},
        # the benchmark's default workload: set-up and solve of the 27-point system, FP32 cycle
        {"name": "poisson27_160_step", "what": "step", "matrix": "poisson27", "nx": 160, "ny": 160, "nz": 160, "cycle": "FP32"},
        # many right-hand sides in time on one matrix, FP64 cycle, no side a power of two
        {"name": "poisson27_ragged_solve", "what": "solve", "matrix": "poisson27", "nx": 127, "ny": 93, "nz": 75, "cycle": "FP64"},
        # the largest: heterogeneous diffusion, values all different, columns beyond int16 offsets
        {"name": "diffusion7_256_step", "what": "step", "matrix": "diffusion7", "nx": 256, "ny": 256, "nz": 256, "cycle": "FP32"},
        # a differentiated solve of an inversion: new matrix values each time, forward and backward
        {"name": "diffusion7_96_grad", "what": "grad", "matrix": "diffusion7", "nx": 96, "ny": 96, "nz": 96, "cycle": "FP32"},
        # 256 uneven systems at once (an ensemble), box sides 10..46
        {"name": "batch256_solve", "what": "batch", "matrix": "poisson7", "m": 256, "lo": 10, "hi": 46, "cycle": "FP32"},
        # 32 right-hand sides through one block solve
        {"name": "poisson27_100_x32", "what": "multi", "matrix": "poisson27", "nx": 100, "ny": 100, "nz": 100, "k": 32, "cycle": "FP32"},
        # one V-cycle as the preconditioner of a user's own loop, heterogeneous values, odd sides
        {"name": "diffusion7_ragged_prec", "what": "prec", "matrix": "diffusion7", "nx": 121, "ny": 101, "nz": 87, "cycle": "FP64"},
        # the settings' other solver and preconditioner: CGHS with l1-Jacobi sweeps
        {"name": "poisson7_64_cghs", "what": "solve", "matrix": "poisson7", "nx": 64, "ny": 64, "nz": 64, "cycle": "FP64",
         "solver": "CGHS", "prec": "L1_JACOBI"},
        # the sparse product on its own, larger than L2
        {"name": "poisson27_160_spmv", "what": "spmv", "matrix": "poisson27", "nx": 160, "ny": 160, "nz": 160},
        # matching on its own, heterogeneous weights
        {"name": "diffusion7_ragged_match", "what": "match", "matrix": "diffusion7", "nx": 75, "ny": 111, "nz": 80},
    ]


#: rows of a drawn case: (fewest, most) by call
_ROWS = {"step": (1e3, 3e6), "solve": (1e3, 3e6), "multi": (1e3, 3e5), "grad": (4e3, 6e5), "prec": (1e3, 3e6), "spmv": (1e3, 6e6),
         "match": (1e3, 2e6)}


def draw(rng):
    what = rng.choice(["step", "step", "solve", "solve", "multi", "batch", "grad", "prec", "spmv", "match"])
    cycle = rng.choice(["FP32", "FP64"])
    if what == "batch":
        lo = rng.randint(8, 20)
        return {"what": "batch", "matrix": "poisson7", "m": rng.randint(3, 64), "lo": lo, "hi": rng.randint(lo + 2, 46), "cycle": cycle}
    matrix = "diffusion7" if what == "grad" else rng.choice(["poisson7", "poisson27", "diffusion7"])
    lo, hi = _ROWS[what]
    rows = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    sx, sy = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
    side = rows ** (1.0 / 3.0)
    nx, ny = max(5, round(side * sx)), max(5, round(side * sy))
    nz = max(5, round(rows / (nx * ny)))
    case = {"what": what, "matrix": matrix, "nx": nx, "ny": ny, "nz": nz}
    if what not in ("spmv", "match"):
        case["cycle"] = cycle
    if what == "multi":
        case["k"] = rng.randint(1, 32)
    if what == "solve" and rng.random() < 0.2 and matrix != "diffusion7":
        case["solver"] = "CGHS"
        case["prec"] = rng.choice(["L1_JACOBI", "BCMG"])
    return case


# ---- inputs -----------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _uniform(n, gen):
    return torch.rand(n, generator=gen, dtype=torch.float64, device=DEV) * 2 - 1


def _kappa(nx, ny, nz, gen):
    """exp(theta): white noise filtered to a Gaussian random field of length 8 and sigma 2, x fastest."""
    w = torch.randn(nz, ny, nx, generator=gen, dtype=torch.float64, device=DEV)
    kz, ky, kx = (2 * math.pi * torch.fft.fftfreq(m, dtype=torch.float64, device=DEV) for m in (nz, ny, nx))
    f = torch.exp(-(kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2) * 8.0 ** 2 / 4)
    th = torch.fft.ifftn(torch.fft.fftn(w) * f).real
    return torch.exp(2.0 * th / torch.sqrt((f ** 2).mean())).reshape(-1)


class _Box:
    """The matrix of a box in 64 bits: its entries by stencil offset, in ascending column order."""

    def __init__(self, matrix, nx, ny, nz, gen, shift=0.0):
        n = nx * ny * nz
        r = torch.arange(n, device=DEV)
        i, j, k = r % nx, (r // nx) % ny, r // (nx * ny)
        full = matrix == "poisson27"
        offs = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
                if full or abs(dx) + abs(dy) + abs(dz) <= 1]
        kap = _kappa(nx, ny, nz, gen) if matrix == "diffusion7" else None
        diag = torch.full((n,), 26.0 if full else 6.0, dtype=torch.float64, device=DEV) + shift
        if kap is not None:
            diag = torch.zeros(n, dtype=torch.float64, device=DEV)
        self.n, self.terms = n, []   # (valid rows, column, value) by offset; None: the diagonal
        for dx, dy, dz in offs:
            if dx == dy == dz == 0:
                self.terms.append(None)
                continue
            ok = (i + dx >= 0) & (i + dx < nx) & (j + dy >= 0) & (j + dy < ny) & (k + dz >= 0) & (k + dz < nz)
            c = torch.where(ok, r + dx + nx * (dy + ny * dz), r)
            if kap is None:
                v = torch.full((n,), -1.0, dtype=torch.float64, device=DEV)
            else:
                t = 2.0 * kap * kap[c] / (kap + kap[c])
                diag = diag + torch.where(ok, t, 2.0 * kap)
                v = -t
            self.terms.append((ok, c.to(torch.int32), v))
        self.diag = diag

    def csr(self):
        cnt = torch.zeros(self.n, dtype=torch.int64, device=DEV)
        for t in self.terms:
            cnt += 1 if t is None else t[0]
        row = torch.zeros(self.n + 1, dtype=torch.int64, device=DEV)
        row[1:] = torch.cumsum(cnt, 0)
        z = int(row[-1])
        at = row[:-1].clone()
        col = torch.empty(z, dtype=torch.int32, device=DEV)
        val = torch.empty(z, dtype=torch.float64, device=DEV)
        ids = torch.arange(self.n, dtype=torch.int32, device=DEV)
        for t in self.terms:
            if t is None:
                col[at], val[at] = ids, self.diag
                at += 1
            else:
                ok, c, v = t
                col[at[ok]], val[at[ok]] = c[ok], v[ok]
                at += ok
        return row.to(torch.int32), col, val

    def times(self, x):
        y = self.diag[:, None] * x if x.dim() == 2 else self.diag * x
        for t in self.terms:
            if t is not None:
                ok, c, v = t
                w = torch.where(ok, v, torch.zeros_like(v))
                y = y + (w[:, None] * x[c.long()] if x.dim() == 2 else w * x[c.long()])
        return y


def _box(case, gen):
    return _Box(case["matrix"], case["nx"], case["ny"], case["nz"], gen)


def _params(case, **kw):
    base = dict(solver=case.get("solver", "FCG"), preconditioner=case.get("prec", "BCMG"), rtol=1e-8, dispnorm=0,
                vcycle_precision=case["cycle"])
    base.update(kw)
    return bx.params_default(**base)


def _batch_boxes(case, seed):
    """The boxes of a batch, the case's own, and their diagonal shifts, the seed's. The batch set-up takes host matrices."""
    g = torch.Generator().manual_seed(case["m"] * 10000 + case["lo"] * 100 + case["hi"])
    dims = torch.randint(case["lo"], case["hi"] + 1, (case["m"], 3), generator=g).tolist()
    g.manual_seed(seed)
    return dims, (0.5 * torch.rand(case["m"], generator=g, dtype=torch.float64)).tolist()


def prepare(case, seed):
    what = case["what"]
    gen = _gen(seed)
    if what == "batch":
        dims, shifts = _batch_boxes(case, seed)
        systems, bs = [], []
        for (nx, ny, nz), shift in zip(dims, shifts):
            A = _Box("poisson7", nx, ny, nz, gen, shift)
            systems.append(tuple(t.cpu().numpy() for t in A.csr()))
            bs.append(A.times(_uniform(A.n, gen)))
        return {"what": what, "batch": bx.Batch(systems, _params(case)), "b": bs}
    A = _box(case, gen)
    row, col, val = A.csr()
    s = {"what": what, "row": row, "col": col, "val": val}
    if what == "spmv":
        s["x"] = _uniform(A.n, gen)
        s["y"] = torch.empty_like(s["x"])
        return s
    if what == "match":
        s["w"] = 0.5 + 0.25 * (_uniform(A.n, gen) + 1)
        return s
    s["params"] = _params(case, rtol=1e-10) if what == "grad" else _params(case)
    if what == "grad":
        s["b"] = A.times(_uniform(A.n, gen))
        s["g"] = A.times(_uniform(A.n, gen))
    elif what == "multi":
        s["b"] = A.times(_uniform(A.n * case["k"], gen).reshape(A.n, case["k"]))
    elif what == "prec":
        s["b"] = _uniform(A.n, gen)
    else:
        s["b"] = A.times(_uniform(A.n, gen))
    if what in ("solve", "multi", "prec"):
        s["h"] = bx.prec_setup(row, col, val, s["params"])
    return s


def run(s):
    what = s["what"]
    if what == "step":
        h = bx.prec_setup(s["row"], s["col"], s["val"], s["params"])
        x, _ = bx.solve(h, s["b"])
        bx.prec_finalize(h)
        return x
    if what == "solve":
        return bx.solve(s["h"], s["b"])[0]
    if what == "multi":
        return s["h"].solve_multi(s["b"])[0]
    if what == "batch":
        xs, _ = s["batch"].solve(s["b"])
        return torch.cat(xs)
    if what == "grad":
        val = s["val"].detach().requires_grad_(True)
        b = s["b"].detach().requires_grad_(True)
        x = autograd.solve(s["row"], s["col"], val, b, s["params"])
        x.backward(s["g"])
        return {"x": x.detach(), "dval": val.grad, "db": b.grad}
    if what == "prec":
        return s["h"].prec_apply(s["b"])
    if what == "spmv":
        return bx.spmv(s["row"], s["col"], s["val"], s["x"], s["y"])
    W, least = bx.edge_weights(s["row"], s["col"], s["val"], s["w"])
    return {"W": W, "least": least, "match": bx.suitor_matching(s["row"], s["col"], W)}


# ---- what a pass cannot do without ------------------------------------------------------------
def _size(matrix, nx, ny, nz):
    n = nx * ny * nz
    if matrix == "poisson27":
        return n, (3 * nx - 2) * (3 * ny - 2) * (3 * nz - 2)
    return n, 7 * n - 2 * (nx * ny + ny * nz + nx * nz)


def _iterations(case):
    """FCG iterations at the case's tolerance, about: constant coefficients grow slowly with the box, the random field's do not."""
    side = (case["nx"] * case["ny"] * case["nz"]) ** (1.0 / 3.0) if "nx" in case else 0.5 * (case["lo"] + case["hi"])
    if case["matrix"] == "diffusion7":
        return 12 * side ** 0.5
    if case.get("prec") == "L1_JACOBI":
        return side
    return 2 * side ** 0.5


def work(case):
    """bytes: the inputs read once, the outputs written once. flops: of a solve, its iterations' products (nine on the finest
    level and its coarser ones' in a cycle, one of the outer iteration); of the others, theirs."""
    what = case["what"]
    if what == "batch":
        side = 0.5 * (case["lo"] + case["hi"])
        n = case["m"] * side ** 3
        return {"bytes": 12 * 7 * n + 20 * n, "flops": _iterations(case) * 2 * 7 * n * (9 * 1.3 + 1)}
    n, z = _size(case["matrix"], case["nx"], case["ny"], case["nz"])
    matrix = 12 * z + 4 * (n + 1)
    if what == "spmv":
        return {"bytes": matrix + 16 * n, "flops": 2 * z}
    if what == "match":
        return {"bytes": matrix + 8 * n + 8 * z + 4 * n, "flops": 8 * z}
    cycle = 2 * z * 9 * (1.15 if case["matrix"] == "poisson27" else 1.5)
    if case.get("prec") == "L1_JACOBI":
        cycle = 2 * z * 3
    if what == "prec":
        return {"bytes": matrix + 16 * n, "flops": cycle}
    iters = _iterations(case) * (1.25 if what == "grad" else 1)
    k = case.get("k", 1)
    flops = iters * (cycle + 2 * z) * k
    if what == "grad":
        return {"bytes": matrix + 32 * n + 8 * z + 8 * n, "flops": 2 * flops}
    return {"bytes": matrix + 16 * n * k, "flops": flops}


def tolerance(case):
    """About four times what was seen. Solves end at a relative residual of 1e-8 (gradients: 1e-10), so two of them that stop an
    iteration apart differ by what is left of the error against x* (6e-7 for the Laplacians, 4e-5 for the largest random field,
    5e-8 for gradients); the other calls differ by the order of their sums (one lane a row against eight: 9e-8 in FP32 cycles,
    with single entries up to 2e-6, and 2e-16 and 4e-15 in FP64 cycles)."""
    what = case["what"]
    if what == "spmv":
        return {"rel": 1e-15, "max": 1e-14}
    if what == "match":
        return {"rel": 1e-15, "max": 1e-14}
    if what == "prec":
        return {"rel": 4e-7, "max": 1e-5} if case["cycle"] == "FP32" else {"rel": 4e-15, "max": 4e-14}
    if what == "grad":
        return {"rel": 2e-7}
    return {"rel": 2e-4 if case["matrix"] == "diffusion7" else 2.5e-6}


def exact(case, seed):
    what = case["what"]
    gen = _gen(seed)
    if what == "batch":
        dims, _ = _batch_boxes(case, seed)
        return torch.cat([_uniform(nx * ny * nz, gen) for nx, ny, nz in dims])
    if what == "prec":
        return None
    A = _box(case, gen)
    if what == "spmv":
        return A.times(_uniform(A.n, gen))
    if what == "multi":
        return _uniform(A.n * case["k"], gen).reshape(A.n, case["k"])
    if what in ("step", "solve"):
        return _uniform(A.n, gen)
    row, col, val = A.csr()
    rows = torch.repeat_interleave(torch.arange(A.n, device=DEV), (row[1:] - row[:-1]).long())
    col = col.long()
    if what == "grad":
        x, lam = _uniform(A.n, gen), _uniform(A.n, gen)
        return {"x": x, "dval": -lam[rows] * x[col], "db": lam}
    w = 0.5 + 0.25 * (_uniform(A.n, gen) + 1)
    off = rows != col
    c = A.diag * w * w
    a = torch.where(off, (1.0 - 2.0 * val * w[rows] * w[col] / (c[rows] + c[col])).abs(), torch.ones_like(val))
    least = float(a[off].min())
    return {"W": torch.log(a), "least": least, "match": None}

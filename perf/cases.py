"""Performance cases of the sparse Krylov path: what a user's program calls, at the sizes of this
repository's workloads (2D Poisson 256^2, 3D anisotropic diffusion 128^3, 3D convection-diffusion 96^3,
2D variable diffusion 512^2, 4,096 Erdos-Renyi Laplacians) and at the small and ragged sizes around them.

A case names a kind of call ("kind"), a matrix ("problem" with its grid nx x ny x nz, natural order, x
fastest) and the call's options.  All inputs are made on the GPU from the seed:

  spmv      A.gemv(trans): the product inside every solver ('T': the adjoint's)
  spmm      A.gemm: one matrix, several right-hand sides
  ilu       M.apply(x, trans): the ILU(0) preconditioner, the largest part of every preconditioned solve
  setup     make_ilu and one apply: what a program pays per new matrix
  cg        solve_cg without a preconditioner (the small 2D systems)
  pcg       solve_cg with ILU(0) in FP64
  ru        solve_ru_pcg: FP32 operator and vectors, FP64 reliable updates
  gmres     solve_gmres with ILU(0) in FP64
  batch     gpu_batch.solve: many independent systems in one call

Solves run to 1e-12 of the right-hand side or tighter, so that their results are the system's solution
to well below their type's rounding bound, whatever the order of a reduction.
"""
import math

import numpy as np
import torch

from hala_gb300 import engine as E

DEV = "cuda"
DTYPES = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16}
_ENGINE = []


def _engine():
    """the program's one engine"""
    if not _ENGINE:
        _ENGINE.append(E.gpu_engine(0))
    return _ENGINE[0]


# ------------------------------------------------------------------------------ the cases ----
def listed():
    return [
        # the smallest call: the preconditioner of a 576-row system (the size of the reference fixtures)
        {"name": "ilu_f64_small", "kind": "ilu", "problem": "poisson2d", "nx": 24, "ny": 24, "nz": 1,
         "store": "f64", "trans": "N"},
        # the FP64 product of the flagship 128^3 system: CG / PCG, residuals and refinement steps
        {"name": "spmv_f64_aniso128", "kind": "spmv", "problem": "aniso3d", "nx": 128, "ny": 128, "nz": 128,
         "dtype": "f64", "trans": "N"},
        # the FP32 product on an unstructured matrix with rows of uneven length (graph Laplacians)
        {"name": "spmv_f32_graph", "kind": "spmv", "problem": "graph", "systems": 701, "nmin": 64, "nmax": 4096,
         "dtype": "f32", "trans": "N"},
        # the transposed product of the adjoint solve on the 512^2 variable-diffusion operator
        {"name": "spmv_f64_t_vardiff512", "kind": "spmv", "problem": "vardiff2d", "nx": 512, "ny": 512, "nz": 1,
         "dtype": "f64", "trans": "T"},
        # several right-hand sides, an odd number of them, on a grid with odd sides
        {"name": "spmm_f32_5rhs", "kind": "spmm", "problem": "convdiff3d", "nx": 95, "ny": 97, "nz": 96,
         "dtype": "f32", "nrhs": 5},
        # the preconditioner of the flagship mixed solve: factor stored in BF16, FP32 vectors
        {"name": "ilu_bf16_aniso128", "kind": "ilu", "problem": "aniso3d", "nx": 128, "ny": 128, "nz": 128,
         "store": "bf16", "trans": "N"},
        # the transposed preconditioner of the adjoint solve on the 512^2 operator, FP32 store
        {"name": "ilu_f32_t_vardiff512", "kind": "ilu", "problem": "vardiff2d", "nx": 512, "ny": 512, "nz": 1,
         "store": "f32", "trans": "T"},
        # a new matrix: the factorisation and the planning of its triangular solves, then one apply
        {"name": "setup_f64_convdiff", "kind": "setup", "problem": "convdiff3d", "nx": 64, "ny": 65, "nz": 61,
         "store": "f64"},
        # a whole small solve: 256^2 Poisson by unpreconditioned CG
        {"name": "cg_poisson256", "kind": "cg", "problem": "poisson2d", "nx": 256, "ny": 256, "nz": 1, "rtol": 1e-13},
        # a whole nonsymmetric solve: 96^3 convection-diffusion by ILU(0)-GMRES(30)
        {"name": "gmres_convdiff96", "kind": "gmres", "problem": "convdiff3d", "nx": 96, "ny": 96, "nz": 96,
         "rtol": 1e-12},
        # many small systems at once: 4,096 graph Laplacians of 64 to 4,096 rows
        {"name": "batch_4096", "kind": "batch", "problem": "graph", "systems": 4096, "nmin": 64, "nmax": 4096,
         "rtol": 1e-12},
        # the flagship whole solve: 128^3 mixed-precision ILU(0)-PCG (the largest case)
        {"name": "ru_pcg_aniso128", "kind": "ru", "problem": "aniso3d", "nx": 128, "ny": 128, "nz": 128,
         "store": "bf16", "rtol": 1e-12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi, dims):
    """grid sides spread around a log-uniform edge, odd ones among them"""
    e = _log(rng, lo, hi)
    s = [max(2, min(hi, int(round(e * rng.uniform(0.8, 1.25))))) for _ in range(dims)]
    return {"nx": s[0], "ny": s[1], "nz": s[2] if dims == 3 else 1}


def _ilu_grid(rng, lo2, hi2, lo3, hi3, free=60000):
    """a grid for an ILU(0) factor: any sides up to `free` rows; above, an x side that is a multiple of
    32, as this repository's large workloads have it"""
    three = hi2 == 0 or rng.random() < 0.5
    m = _grid(rng, lo3, hi3, 3) if three else _grid(rng, lo2, hi2, 2)
    if m["nx"] * m["ny"] * m["nz"] > free:
        m["nx"] = max(32, m["nx"] // 32 * 32)
    return m


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmm", "ilu", "ilu", "ilu", "setup", "cg", "pcg", "ru", "gmres", "batch"])
    graph = {"problem": "graph", "systems": _log(rng, 60, 4096), "nmin": rng.choice([64, 100]),
             "nmax": rng.choice([500, 2000, 4096])}
    two = {"problem": rng.choice(["poisson2d", "vardiff2d"])}
    three = {"problem": rng.choice(["aniso3d", "convdiff3d"])}
    if kind in ("spmv", "spmm"):
        m = rng.choice([graph, {**two, **_grid(rng, 200, 768, 2)}, {**three, **_grid(rng, 36, 128, 3)}])
        if kind == "spmm":
            return {"kind": kind, **m, "dtype": rng.choice(["f64", "f32"]), "nrhs": rng.randint(2, 9)}
        dt = rng.choice(["f64", "f64", "f32", "f32", "bf16"])
        return {"kind": kind, **m, "dtype": dt, "trans": "N" if dt == "bf16" else rng.choice(["N", "N", "T"])}
    if kind == "ilu":
        m = _ilu_grid(rng, 16, 512, 8, 128)
        m = {**(three if m["nz"] > 1 else two), **m}
        return {"kind": kind, **m, "store": rng.choice(["f64", "f32", "bf16"]), "trans": rng.choice(["N", "N", "T"])}
    if kind == "setup":
        m = _ilu_grid(rng, 16, 320, 8, 80, free=20000)
        m = {**(three if m["nz"] > 1 else two), **m}
        return {"kind": kind, **m, "store": rng.choice(["f64", "f32", "bf16"])}
    if kind == "cg":
        return {"kind": kind, "problem": "poisson2d", **_grid(rng, 16, 300, 2), "rtol": 1e-13}
    if kind == "pcg":
        return {"kind": kind, "problem": "aniso3d", **_ilu_grid(rng, 0, 0, 10, 88, 3), "rtol": 1e-12}
    if kind == "ru":
        return {"kind": kind, "problem": "aniso3d", **_ilu_grid(rng, 0, 0, 10, 110, 3), "store": rng.choice(["f32", "bf16"]),
                "rtol": 1e-12}
    if kind == "gmres":
        return {"kind": kind, "problem": "convdiff3d", **_ilu_grid(rng, 0, 0, 10, 96, 3), "rtol": 1e-12}
    return {"kind": "batch", **graph, "rtol": 1e-12}


# ---------------------------------------------------------------------------- the matrices ----
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _stencil(case):
    """(axis, direction, constant value) of the off-diagonals in ascending column order, and the diagonal"""
    p = case["problem"]
    if p == "poisson2d":
        return [(1, -1, -1.0), (0, -1, -1.0), (None, 0, 4.0), (0, 1, -1.0), (1, 1, -1.0)]
    if p == "aniso3d":
        c = (1.0, 1.0, 0.01)
        off = [(a, -1, -c[a]) for a in (2, 1, 0)] + [(None, 0, 2.0 * sum(c))] + [(a, 1, -c[a]) for a in (0, 1, 2)]
        return off
    assert p == "convdiff3d"      # velocity (1, 0.5, 0.25), cell Peclet number 10, first-order upwind
    up = (10.0, 5.0, 2.5)
    return ([(a, -1, -1.0 - up[a]) for a in (2, 1, 0)] + [(None, 0, 6.0 + sum(up))] +
            [(a, 1, -1.0) for a in (0, 1, 2)])


def _grid_entries(case, g):
    """[n, k] value and validity arrays of the grid operator and its k column offsets (float64, GPU)"""
    shape = (case["nx"], case["ny"], case["nz"])
    stride = (1, shape[0], shape[0] * shape[1])
    n = shape[0] * shape[1] * shape[2]
    rows = torch.arange(n, device=DEV)
    xyz = (rows % shape[0], (rows // shape[0]) % shape[1], rows // (shape[0] * shape[1]))
    ok, val, off = [], [], []
    if case["problem"] == "vardiff2d":
        nx, ny = shape[0], shape[1]
        # cell conductivities exp(Gaussian random field of correlation length 16, sigma 1); harmonic-mean
        # faces, 2 k at the Dirichlet boundary
        fx = torch.fft.fftfreq(nx, device=DEV, dtype=torch.float64)
        fy = torch.fft.fftfreq(ny, device=DEV, dtype=torch.float64)
        spec = torch.exp(-(2 * math.pi * 16.0) ** 2 * (fx[None, :] ** 2 + fy[:, None] ** 2) / 2)
        w = torch.randn(ny, nx, device=DEV, dtype=torch.float64, generator=g)
        f = torch.fft.ifft2(torch.fft.fft2(w) * spec.sqrt()).real
        k = torch.exp((f - f.mean()) / f.std().clamp_min(1e-12))
        kx = torch.empty(ny, nx + 1, device=DEV, dtype=torch.float64)
        ky = torch.empty(ny + 1, nx, device=DEV, dtype=torch.float64)
        kx[:, 1:-1] = 2 * k[:, :-1] * k[:, 1:] / (k[:, :-1] + k[:, 1:])
        kx[:, 0], kx[:, -1] = 2 * k[:, 0], 2 * k[:, -1]
        ky[1:-1] = 2 * k[:-1] * k[1:] / (k[:-1] + k[1:])
        ky[0], ky[-1] = 2 * k[0], 2 * k[-1]
        w_, e_, s_, n_ = (t.reshape(-1) for t in (kx[:, :-1], kx[:, 1:], ky[:-1], ky[1:]))
        terms = [(1, -1, -s_), (0, -1, -w_), (None, 0, w_ + e_ + s_ + n_), (0, 1, -e_), (1, 1, -n_)]
    else:
        terms = _stencil(case)
    for axis, d, v in terms:
        if axis is None:
            ok.append(torch.ones(n, dtype=torch.bool, device=DEV))
            off.append(0)
        else:
            c = xyz[axis] + d
            ok.append((c >= 0) & (c < shape[axis]))
            off.append(d * stride[axis])
        val.append(v if isinstance(v, torch.Tensor) else torch.full((n,), v, device=DEV, dtype=torch.float64))
    val, ok = torch.stack(val, 1), torch.stack(ok, 1)
    if case["kind"] == "setup":     # a reaction term of the seed's own: another matrix for each seed
        val[:, off.index(0)] += torch.rand(n, device=DEV, dtype=torch.float64, generator=g)
    return val, ok, off


def _sizes(case):
    u = (torch.arange(case["systems"], device=DEV, dtype=torch.float64) + 0.5) / case["systems"]
    return torch.exp(math.log(case["nmin"]) + u * math.log(case["nmax"] / case["nmin"])).long()


def _csr(case, g):
    """(pntr, indx, float64 vals, sys_ptr or None)"""
    if case["problem"] != "graph":
        val, ok, off = _grid_entries(case, g)
        n = val.shape[0]
        cols = torch.arange(n, device=DEV)[:, None] + torch.tensor(off, device=DEV)[None, :]
        pntr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
        pntr[1:] = torch.cumsum(ok.sum(1), 0)
        return pntr, cols[ok].to(torch.int32), val[ok].contiguous(), None
    # independent Erdos-Renyi graph Laplacians (mean degree 8, weights in [0.1, 1)) + 0.01 I, block-diagonal
    # with global columns; the sizes (log-uniform, in the seed's order) are the case's own
    size = _sizes(case)[torch.randperm(case["systems"], device=DEV, generator=g)]
    sys_ptr = torch.zeros(case["systems"] + 1, dtype=torch.int64, device=DEV)
    sys_ptr[1:] = torch.cumsum(size, 0)
    n, count = int(sys_ptr[-1]), case["systems"]
    s = torch.repeat_interleave(torch.arange(count, device=DEV), size * 4)   # 4 n edges: mean degree 8
    m = size[s]
    a = (torch.rand(len(s), device=DEV, generator=g, dtype=torch.float64) * m).long()
    b = (torch.rand(len(s), device=DEV, generator=g, dtype=torch.float64) * m).long()
    keep = a != b
    a, b, base = a[keep], b[keep], sys_ptr[s[keep]]
    key = torch.unique((base + torch.minimum(a, b)) * n + base + torch.maximum(a, b))
    r, c = key // n, key % n
    w = 0.1 + 0.9 * torch.rand(len(key), device=DEV, generator=g, dtype=torch.float64)
    order = torch.argsort(torch.cat([key, c * n + r, torch.arange(n, device=DEV) * (n + 1)]))
    rows = torch.cat([r, c, torch.arange(n, device=DEV)])[order]
    cols = torch.cat([c, r, torch.arange(n, device=DEV)])[order]
    vals = torch.cat([-w, -w, torch.zeros(n, device=DEV, dtype=torch.float64)])[order]
    pntr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    pntr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    vals = vals.float().double()      # the batch holds FP32 values: the diagonal sums those
    total = torch.cat([torch.zeros(1, device=DEV, dtype=torch.float64), torch.cumsum(vals, 0)])
    diag = rows == cols
    vals[diag] = (0.01 - (total[pntr[1:]] - total[pntr[:-1]])).float().double()
    return pntr.to(torch.int32), cols.to(torch.int32), vals.contiguous(), sys_ptr.to(torch.int32)


def _product(pntr, indx, vals, x):
    """A x in float64 (plain torch)"""
    return torch.segment_reduce(vals.double() * x.double()[indx.long()], "sum",
                                lengths=(pntr[1:] - pntr[:-1]).long())


def _product_t(pntr, indx, vals, x):
    n = pntr.numel() - 1
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (pntr[1:] - pntr[:-1]).long())
    return torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, indx.long(), vals.double() * x.double()[rows])


# ------------------------------------------------------------------------ prepare and run ----
def _inputs(case, seed):
    """the matrix and the vectors of a case: everything but the handles"""
    g = _gen(seed)
    pntr, indx, vals, sys_ptr = _csr(case, g)
    n = pntr.numel() - 1
    k = case["kind"]
    s = {"pntr": pntr, "indx": indx, "vals": vals, "sys_ptr": sys_ptr, "n": n}
    if k in ("spmv", "spmm"):
        dt = DTYPES[case["dtype"]]
        s["vals"] = vals.to(dt)
        xdt = torch.float64 if dt == torch.float64 else torch.float32
        shape = (n,) if k == "spmv" else (case["nrhs"], n)      # column-major: a row here is a column
        s["x"] = torch.randn(shape, device=DEV, dtype=torch.float64, generator=g).to(xdt)
    elif k in ("ilu", "setup"):
        xdt = torch.float64 if case["store"] == "f64" else torch.float32
        s["x"] = torch.randn(n, device=DEV, dtype=torch.float64, generator=g).to(xdt)
    else:      # solves: b = A x_true
        s["x_true"] = torch.randn(n, device=DEV, dtype=torch.float64, generator=g)
        s["b"] = _product(pntr, indx, vals, s["x_true"])
    return s


def prepare(case, seed):
    eng = _engine()
    s = _inputs(case, seed)
    k, n, p, i, v = case["kind"], s["n"], s["pntr"], s["indx"], s["vals"]
    s.update(kind=k, case=case, eng=eng)
    if k in ("spmv", "spmm"):
        s["A"] = E.make_sparse_matrix(eng, n, p, i, v)
        s["y"] = torch.empty_like(s["x"])
    elif k == "ilu":
        s["M"] = E.make_ilu(eng, p, i, v, store=DTYPES[case["store"]])
        s["r"] = torch.empty_like(s["x"])
    elif k in ("cg", "pcg", "gmres"):
        s["A"] = E.make_sparse_matrix(eng, n, p, i, v)
        s["M"] = E.make_ilu(eng, p, i, v) if k != "cg" else None
        norm = (s["M"].apply(s["b"]) if k == "gmres" else s["b"]).norm().item()
        s["stop"] = E.stop_criteria(case["rtol"] * norm, 100000 if k != "gmres" else 1000)
    elif k == "ru":
        s["A"] = E.make_sparse_matrix(eng, n, p, i, v)
        s["vals32"] = v.float()
        s["A32"] = E.make_sparse_matrix(eng, n, p, i, s["vals32"])
        s["M"] = E.make_ilu(eng, p, i, v, store=DTYPES[case["store"]])
        s["tol"] = case["rtol"] * s["b"].norm().item()
    elif k == "batch":
        s["vals32"] = v.float()
        s["batch"] = E.gpu_batch(eng, s["sys_ptr"], p, i, s["vals32"])
    return s


def run(s):
    k = s["kind"]
    if k == "spmv":
        return s["A"].gemv(s["case"]["trans"], 1.0, s["x"], 0.0, s["y"])
    if k == "spmm":
        return s["A"].gemm(s["case"]["nrhs"], 1.0, s["x"], 0.0, s["y"])
    if k == "ilu":
        return s["M"].apply(s["x"], s["r"], s["case"]["trans"])
    if k == "setup":
        M = E.make_ilu(s["eng"], s["pntr"], s["indx"], s["vals"], store=DTYPES[s["case"]["store"]])
        factor, diag = M.factor()
        return {"factor": factor, "diag": diag, "r": M.apply(s["x"])}
    x = torch.zeros(s["n"], dtype=torch.float64, device=DEV)
    if k in ("cg", "pcg"):
        E.solve_cg(s["eng"], s["stop"], s["pntr"], s["indx"], s["vals"], s["b"], x, ilu=s["M"], matrix=s["A"])
    elif k == "gmres":
        E.solve_gmres(s["eng"], s["stop"], 30, s["pntr"], s["indx"], s["vals"], s["b"], x, ilu=s["M"], matrix=s["A"])
    elif k == "ru":
        E.solve_ru_pcg(s["eng"], s["A"], s["A32"], s["M"], s["b"], x, s["tol"])
    else:
        s["batch"].solve(s["b"], x, rtol=s["case"]["rtol"])
    return x


# ------------------------------------------------------------------------------- the work ----
def work(case):
    k = case["kind"]
    if case["problem"] == "graph":
        lo, hi = case["nmin"], case["nmax"]
        n = case["systems"] * (hi - lo) / math.log(hi / lo)
        nnz = 9 * n
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        nnz = n + 2 * (n - n // nx) + 2 * (n - n // ny) + (2 * (n - n // nz) if nz > 1 else 0)
    size = {"f64": 8, "f32": 4, "bf16": 2}
    if k in ("spmv", "spmm"):
        vs, xs = size[case["dtype"]], 8 if case["dtype"] == "f64" else 4
        m = case.get("nrhs", 1)
        return {"bytes": nnz * (vs + 4) + 4 * n + 2 * xs * n * m, "flops": 2 * nnz * m}
    if k in ("ilu", "setup"):
        vs, xs = size[case["store"]], 8 if case["store"] == "f64" else 4
        apply = nnz * (vs + 4) + 4 * n + 2 * xs * n + (8 * n if vs < 8 else 0)
        if k == "ilu":
            return {"bytes": apply, "flops": 2 * nnz}
        # the matrix read, the factor and the diagonal index written, the apply; two flops per update
        return {"bytes": nnz * 20 + 8 * n + apply, "flops": 5 * nnz}
    # solves: the matrix and b read once, x written once; the operations of every iteration, with the
    # iteration counts that these operators take
    io = nnz * 12 + 4 * n + 16 * n
    if k == "cg":
        its = 3.9 * (nx + ny) / 2
        return {"bytes": io, "flops": its * (2 * nnz + 10 * n)}
    if k in ("pcg", "ru"):
        its = 8 + 1.55 * (nx + ny) / 2
        return {"bytes": io, "flops": its * (4 * nnz + 12 * n)}
    if k == "gmres":
        its = 10 + 0.28 * (nx + ny + nz) / 3
        return {"bytes": io, "flops": its * (4 * nnz + 4 * n * min(its, 30) / 2)}
    return {"bytes": nnz * 8 + 4 * n + 16 * n, "flops": 170 * (2 * nnz + 10 * n)}


# ---------------------------------------------------------------- the results in 64 bits ----
def _levels(case):
    """the rows of a grid by x + y + z: row sets that do not depend on one another"""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.arange(nx * ny * nz)
    lev = r % nx + (r // nx) % ny + r // (nx * ny)
    order = np.argsort(lev, kind="stable")
    return np.split(order, np.cumsum(np.bincount(lev))[:-1])


def _exact_ilu(case, seed):
    """ILU(0) of the grid operator, level by level: no two neighbours of a grid point are neighbours
    of each other, so only the diagonal changes.  Returns ([n, k] factor, validity, offsets, levels)."""
    val, ok, off = _grid_entries(case, _gen(seed))
    f, ok = val.cpu().numpy().copy(), ok.cpu().numpy()
    d, low = off.index(0), [q for q, o in enumerate(off) if o < 0]
    levels = _levels(case)
    for rows in levels:
        for q in low:
            r = rows[ok[rows, q]]
            c = r + off[q]
            f[r, q] /= f[c, d]
            f[r, d] -= f[r, q] * f[c, off.index(-off[q])]
    return f, ok, off, levels


def _exact_apply(f, ok, off, levels, x, trans):
    d = off.index(0)
    low, upp = [q for q, o in enumerate(off) if o < 0], [q for q, o in enumerate(off) if o > 0]
    y = x.astype(np.float64).copy()
    for rows in levels:      # L y = x, or U^T y = x
        for q in low:
            r = rows[ok[rows, q]]
            c = r + off[q]
            y[r] -= (f[r, q] if trans == "N" else f[c, off.index(-off[q])]) * y[c]
        if trans != "N":
            y[rows] /= f[rows, d]
    for rows in reversed(levels):      # U r = y, or L^T r = y
        for q in upp:
            r = rows[ok[rows, q]]
            c = r + off[q]
            y[r] -= (f[r, q] if trans == "N" else f[c, off.index(-off[q])]) * y[c]
        if trans == "N":
            y[rows] /= f[rows, d]
    return y


def exact(case, seed):
    k = case["kind"]
    s = _inputs(case, seed)
    if k == "spmv":
        f = _product if case["trans"] == "N" else _product_t
        return f(s["pntr"], s["indx"], s["vals"], s["x"])
    if k == "spmm":
        return torch.stack([_product(s["pntr"], s["indx"], s["vals"], c) for c in s["x"]])
    if k in ("ilu", "setup"):
        f, ok, off, levels = _exact_ilu(case, seed)
        r = _exact_apply(f, ok, off, levels, s["x"].cpu().numpy(), case.get("trans", "N"))
        return r if k == "ilu" else {"factor": f[ok], "diag": None, "r": r}
    return s["x_true"]

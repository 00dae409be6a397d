"""ILU(0) applications on both sides of the choice between strips and levels, FP64 and FP32, 'N' and 'T', bit for bit the
oracle's: grids of which some rows have more than three entries in a triangle (strips, their entries listed apart), random and
reordered patterns, wide stencils, chains, a triangular matrix (one sweep without levels)."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.csgraph as csgraph
import torch

from hala_gb300 import engine as E
from hala_gb300 import problems as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def matrix(f):
    p, i, v = f
    return sp.csr_matrix((v, i, p))


def couple(A, count, rng):
    """some symmetric couplings between rows at most 3000 apart"""
    n = A.shape[0]
    r = rng.integers(0, n - 3000, count)
    c = r + rng.integers(2, 3000, count)
    B = sp.coo_matrix((rng.uniform(-0.1, 0.1, count), (r, c)), shape=(n, n))
    return A + B + B.T


def reorder(A, q):
    return A[q][:, q]


def offsets(n, distances, rng):
    B = sp.diags([rng.uniform(-1, 1, n - d) for d in distances], [-d for d in distances])
    return B + B.T


def stencil(nx, ny, nz, rng):
    n = nx * ny * nz
    i = np.arange(n)
    x, y, z = i % nx, i // nx % ny, i // (nx * ny)
    r, c = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0) & (z + dz < nz)
                r.append(i[ok])
                c.append(i[ok] + dx + nx * dy + nx * ny * dz)
    r, c = np.concatenate(r), np.concatenate(c)
    return sp.csr_matrix((rng.uniform(-1, 1, len(r)), (r, c)), shape=(n, n))


CASES = {
    "grid_some_long_rows": lambda g: couple(matrix(P.poisson2d(301, 97)), 200, g),
    "grid3d_some_long_rows": lambda g: couple(matrix(P.aniso3d(64, 65, 9)), 60, g),
    "grid_permuted": lambda g: reorder(matrix(P.aniso3d(20, 20, 20)), g.permutation(8000)),
    "grid_rcm": lambda g: reorder(matrix(P.aniso3d(30, 30, 30)), csgraph.reverse_cuthill_mckee(matrix(P.aniso3d(30, 30, 30)), True)),
    "random_20000_3": lambda g: sp.random(20000, 20000, 1.5 / 20000, random_state=1),
    "path_permuted": lambda g: reorder(sp.csr_matrix(offsets(20000, [1], g)), g.permutation(20000)),
    "stencil27": lambda g: stencil(17, 16, 15, g),
    "stencil9": lambda g: stencil(60, 59, 1, g),
    "band_5": lambda g: offsets(3000, [1, 2, 3, 4, 5], g),
    "upper_triangle": lambda g: sp.triu(offsets(3000, [1, 7], g)),
    "lower_triangle": lambda g: sp.tril(offsets(3000, [1, 2, 3, 4, 9], g)),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_apply_bit_exact(eng, rng, name, dtype):
    A = sp.csr_matrix(CASES[name](rng))
    A = sp.csr_matrix(A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 1.0 - A.diagonal()))
    A.sort_indices()
    n = A.shape[0]
    p, i, v = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data.astype(np.float64 if dtype == torch.float64 else np.float32)
    fo, do, _ = O.ilu_factor(p, i, v)
    M = E.make_ilu(eng, T(p), T(i), T(v))
    for k in range(2):
        x = rng.standard_normal(n).astype(v.dtype)
        for trans in "NT":
            assert np.array_equal(M.apply(T(x), trans=trans).cpu().numpy(), O.ilu_apply(p, i, do, fo, x, trans=trans)), (k, trans)
    for uplo in "LU":      # the level sets, whichever schedule the applications take
        lev, nl = M.levels(uplo)
        lo, nlo = O.levels(p, i, do, uplo)
        assert nl == nlo and np.array_equal(lev.cpu().numpy(), lo)


@pytest.mark.parametrize("name", ["grid_some_long_rows", "grid_permuted"])
@pytest.mark.parametrize("host", [False, True])
def test_mixed_store_bit_exact(eng, rng, name, host):
    """an FP64 factor stored in FP32 (FP64 pivots), from device and from host buffers, by strips and by levels"""
    A = sp.csr_matrix(CASES[name](rng))
    A = sp.csr_matrix(A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 1.0 - A.diagonal()))
    A.sort_indices()
    p, i, v = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    fo, do, _ = O.ilu_factor(p, i, v)
    M = E.make_ilu_host(eng, p, i, v, store=torch.float32) if host else E.make_ilu(eng, T(p), T(i), T(v), store=torch.float32)
    for _ in range(2):
        x = rng.standard_normal(A.shape[0]).astype(np.float32)
        assert np.array_equal(M.apply(T(x)).cpu().numpy(), O.ilu_apply_mixed(p, i, do, fo.astype(np.float32), fo[do], x))


def test_solves_by_levels(eng, rng):
    """whole solves (graph replay, launches after the end as no-ops) with a preconditioner applied by levels"""
    A = reorder(matrix(P.aniso3d(24, 23, 22)), rng.permutation(24 * 23 * 22))
    A.sort_indices()
    n = A.shape[0]
    p, i, v = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    xt = rng.standard_normal(n)
    b = A @ xt
    tol = 1e-10 * np.linalg.norm(b)
    fo, do, _ = O.ilu_factor(p, i, v)
    _, ito, _ = O.cg(p, i, v, b, tol=tol, diag=do, ilu=fo)
    a = [T(p), T(i), T(v)]
    A64 = E.make_sparse_matrix(eng, n, *a)
    for trans in "NT":
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        info = E.solve_cg_op(eng, A64, E.make_ilu(eng, *a), trans, T(b), x, tol, max_iter=5000)
        assert abs(info.iterations - ito) <= max(1, ito // 20)
        assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01 * tol
    A32 = E.make_sparse_matrix(eng, n, a[0], a[1], a[2].float())
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    info = E.solve_ru_pcg(eng, A64, A32, E.make_ilu(eng, *a, store=torch.bfloat16), T(b), x, tol, delta=0.01)
    assert np.linalg.norm(b - A @ x.cpu().numpy()) <= 1.01 * tol and info.iterations <= 1.1 * ito + 2

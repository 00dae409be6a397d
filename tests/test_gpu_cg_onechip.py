"""The persistent CG at the edges of its launch shapes: one row, a CTA's rows and one more, the largest systems
of one, two and four rows per thread and the first beyond each, rows longer than a thread keeps in registers, empty
off-diagonals, more iterations than one launch runs.  The matrix is a weighted graph Laplacian plus the identity
(symmetric, smallest eigenvalue 1): two solutions to a residual of tol differ by at most 2 tol, and the general
path is the same call with the transposed operator."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E

pytestmark = pytest.mark.gpu


def system(n, reach, seed):
    """off-diagonals at the given distances (their entries dropped at random), diagonal 1 + the row's weights"""
    rng = np.random.default_rng(seed)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.ones(n)]
    for d in reach:
        i = np.arange(n - d) if d < n else np.zeros(0, int)
        i = i[rng.random(len(i)) < 0.9]
        w = rng.uniform(0.1, 1.0, len(i))
        rows += [i, i + d, i, i + d]
        cols += [i + d, i, i, i + d]
        vals += [-w, -w, w, w]
    import scipy.sparse as sp
    A = sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), shape=(n, n))
    A.sum_duplicates()
    A.sort_indices()
    return A, rng


def solve(A, b, dtype, rtol, trans, mode="fused"):
    eng = E.gpu_engine(0)
    eng.set_spmv_mode(mode)
    dev = [torch.tensor(a).cuda() for a in (A.indptr.astype(np.int32), A.indices.astype(np.int32))]
    M = E.make_sparse_matrix(eng, A.shape[0], *dev, torch.tensor(A.data).to(dtype).cuda())
    vt = torch.float64 if dtype == torch.float64 else torch.float32
    x = torch.zeros(A.shape[0], dtype=vt, device="cuda")
    tol = rtol * np.linalg.norm(b)
    info = E.solve_cg_op(eng, M, None, trans, torch.tensor(b).to(vt).cuda(), x, tol, max_iter=20000)
    return x.cpu().numpy().astype(np.float64), info


GRID = [1, 70]
SIZES = [(1, GRID), (2, [1]), (255, GRID), (256, GRID), (257, GRID), (2048, GRID), (2049, [1, 300]), (38912, [1, 200]), (38913, [1, 200]),
         (77824, [1, 256, 60000]), (77825, [1, 256]), (155648, [1, 400]), (155649, [1, 400]), (36864, [1, 200]), (36865, [1, 200]), (73728, [1, 256]), (73729, [1, 256]), (147456, [1, 400]), (147457, [1, 400]),
          (5000, [1, 2, 3, 40, 1000]), (40001, [1, 2, 7, 9000, 30000])]


@pytest.mark.parametrize("dtype,rtol", [(torch.float64, 1e-11), (torch.float32, 1e-4)])
@pytest.mark.parametrize("n,reach", SIZES)
def test_same_solution_as_the_general_path(n, reach, dtype, rtol):
    A, rng = system(n, reach, n)
    if dtype == torch.float32:
        A.data = A.data.astype(np.float32).astype(np.float64)
    b = rng.standard_normal(n)
    if dtype == torch.float32:
        b = b.astype(np.float32).astype(np.float64)
    tol = rtol * np.linalg.norm(b)
    for mode in ("fused", "exact"):
        x, info = solve(A, b, dtype, rtol, "N", mode)
        y, ref = solve(A, b, dtype, rtol, "T", mode)
        assert np.linalg.norm(b - A @ x) <= 2 * tol
        assert np.linalg.norm(x - y) <= 4 * tol
        assert abs(info.iterations - ref.iterations) <= 2 + ref.iterations // 20


def test_more_iterations_than_one_launch():
    """a chain whose exact solution takes as many steps as rows: the direction carries over between launches"""
    import scipy.sparse as sp
    n = 6000
    A = sp.diags([-np.ones(n - 1), np.full(n, 2.0), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    b = np.zeros(n)
    b[0] = 1.0
    x, info = solve(A, b, torch.float64, 1e-8, "N")
    assert info.iterations > 4096
    assert np.linalg.norm(b - A @ x) <= 2e-8

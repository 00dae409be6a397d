"""The batch's on-chip systems at the edges of their shapes (512, 1024, 2048 and 4096 rows), next to systems that
do not fit (a row with more than 255 off-diagonal entries), single rows, diagonal systems, a start other
than zero and right-hand sides whose squares are outside FP32's range.  Every system has to meet its
residual target, measured in FP64, and agree with a dense FP64 solve to the target times the condition
number's bound (shift 0.01 against a largest eigenvalue below 2 max_i a_ii)."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from hala_gb300 import problems as P

pytestmark = pytest.mark.gpu
dev = torch.device("cuda")


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def star(n, shift=0.01):
    """a hub with n - 1 leaves: the hub's row holds every column"""
    A = np.zeros((n, n))
    A[0, 1:] = A[1:, 0] = -0.25
    np.fill_diagonal(A, -A.sum(1) + shift)
    return A


def csr(A):
    r, c = np.nonzero(A)
    p = np.zeros(len(A) + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=len(A)), out=p[1:])
    return p, c.astype(np.int64), A[r, c]


def system(kind, n, rng):
    if kind == "star":
        return csr(star(n))
    if kind == "diag":
        return np.arange(n + 1), np.arange(n), rng.uniform(1, 2, n)
    return P.er_laplacian(n, rng)


BATCHES = {
    "edges": [("er", n) for n in (1, 2, 31, 32, 33, 511, 512, 513, 1024, 1025, 2048, 2049, 4095, 4096)],
    "rows_too_long": [("star", 256), ("star", 257), ("star", 700), ("er", 300), ("star", 3000), ("diag", 40)],
    "diagonal": [("diag", 1), ("diag", 64), ("diag", 4096), ("er", 100)],
    "one": [("er", 777)],
}


@pytest.mark.parametrize("name", list(BATCHES))
@pytest.mark.parametrize("scale", [1.0, 1e-28, 1e24])
def test_onchip_batch(eng, name, scale):
    rng = np.random.default_rng(11)
    sp, P_, I, V = [0], [np.zeros(1, np.int64)], [], []
    for kind, n in BATCHES[name]:
        p, i, v = system(kind, n, rng)
        P_.append(p[1:] + P_[-1][-1])
        I.append(i + sp[-1])
        V.append(v)
        sp.append(sp[-1] + n)
    p, i, v = np.concatenate(P_).astype(np.int32), np.concatenate(I).astype(np.int32), np.concatenate(V).astype(np.float32)
    b = rng.standard_normal(sp[-1]) * scale
    x0 = rng.standard_normal(sp[-1]) * scale
    B = E.gpu_batch(eng, T(np.array(sp, np.int32)), T(p), T(i), T(v))
    rel = torch.zeros(len(sp) - 1, dtype=torch.float64, device=dev)
    its = torch.zeros(len(sp) - 1, dtype=torch.int32, device=dev)
    x, again = T(x0), T(x0)
    B.solve(T(b), x, rtol=1e-11, iters=its, relres=rel)
    B.solve(T(b), again, rtol=1e-11)
    assert torch.equal(x, again)      # the same bits in every run
    xs = x.cpu().numpy()
    v64 = v.astype(np.float64)
    r = b - P.csr_matvec(p, i, v64, xs)
    for s, (kind, n) in enumerate(BATCHES[name]):
        q = slice(sp[s], sp[s + 1])
        assert np.linalg.norm(r[q]) <= 1.01e-11 * np.linalg.norm(b[q]), (s, kind, n)
        if n <= 1100:
            ps = p[sp[s]:sp[s + 1] + 1] - p[sp[s]]
            e = slice(p[sp[s]], p[sp[s + 1]])
            A = P.csr_to_dense(ps, i[e] - sp[s], v64[e])
            xo = np.linalg.solve(A, b[q])
            cond = 2 * A.diagonal().max() / 0.005
            assert np.linalg.norm(xs[q] - xo) <= 1e-11 * cond * np.linalg.norm(xo) * 2, (s, kind, n)
    assert np.all(rel.cpu().numpy() <= 1e-11) and np.all(its.cpu().numpy() >= 1)

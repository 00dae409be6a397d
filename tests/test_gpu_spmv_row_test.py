"""The products around the 64 entries from which a matrix handle compiles the long-row test in, and without a handle,
where the rows' lengths are not known: the bits of the unstaged kernel."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E

pytestmark = pytest.mark.gpu
DT = {"f64": (torch.float64, torch.float64), "f32": (torch.float32, torch.float32), "bf16": (torch.bfloat16, torch.float32)}


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("short,longest", [(7, 7), (7, 63), (7, 64), (0, 63), (9, 300), (11, 65)])
def test_longest_row(short, longest, dtype):
    eng = E.gpu_engine(0)
    vt, xt = DT[dtype]
    n = 3001
    rng = np.random.default_rng(longest)
    ln = np.full(n, short)
    ln[5:n:61] = longest
    ln[8:40] = max(short, 9)      # a tile that is not staged
    ln[n - 1] = longest
    pntr = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    at = np.arange(pntr[-1]) - np.repeat(pntr[:-1], ln)
    indx = (np.repeat(rng.integers(0, n - 8 * longest, n), ln) + 8 * at).astype(np.int32)
    p, i = torch.tensor(pntr).cuda(), torch.tensor(indx).cuda()
    v = torch.tensor(rng.standard_normal(len(indx))).to(vt).cuda()
    x = torch.tensor(rng.standard_normal((3, n))).to(xt).cuda()
    y0 = torch.tensor(rng.standard_normal((3, n))).to(xt).cuda()
    u = torch.empty(len(indx) + 1, dtype=vt, device="cuda")[1:]
    u.copy_(v)
    A, B = E.make_sparse_matrix(eng, n, p, i, v), E.make_sparse_matrix(eng, n, p, i, u)
    for mode in ("fused", "exact"):
        eng.set_spmv_mode(mode)
        for alpha, beta in ((1.0, 0.0), (1.5, -2.0)):
            ref, y, z, m = (y0.clone() for _ in range(4))
            for c in range(3):
                B.gemv("N", alpha, x[c], beta, ref[c])
                A.gemv("N", alpha, x[c], beta, y[c])
                E.sparse_gemv(eng, "N", n, n, alpha, p, i, v, x[c], beta, z[c])
            A.gemm(3, alpha, x, beta, m)
            assert torch.equal(y, ref) and torch.equal(z, ref) and torch.equal(m, ref), (mode, alpha)

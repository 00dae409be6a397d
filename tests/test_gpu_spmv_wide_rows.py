"""Products with long rows among short ones: in fused and exact mode, at every (alpha, beta) form and for several columns,
the bits of the unstaged kernel (the route of arrays that are not 16-byte aligned); in exact mode the oracle's.  Row lengths
around the 64 entries from which a row is summed by its warp, its chunks of 32, and the shares of a tile (a third, an
eighth) up to which it is; long rows in the last, partial tile; several tiles per warp, staged and not, in one matrix."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DT = {"f64": (torch.float64, torch.float64), "f32": (torch.float32, torch.float32), "bf16": (torch.bfloat16, torch.float32)}


def unaligned(t):
    """the same values at an address that is not a multiple of 16 bytes"""
    u = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:]
    u.copy_(t)
    assert u.data_ptr() % 16
    return u


# rows, short rows' lengths, {row: length}
SHAPES = [(700, [0], {0: 257, 33: 288, 95: 289, 699: 700}),
          (4000, [6], {5: 63, 40: 64, 70: 65, 100: 1000, 131: 3001, 3999: 4000}),
          (3001, [5, 0, 7], {1: 2000, 2: 700, 3: 700, 4: 100, 64: 900, 65: 900, 66: 900, 67: 900, 3000: 1500}),
          (2000, [30], {7: 479, 40: 480, 70: 481, 100: 135, 133: 140, 1999: 1025}),
          (1000, [80], {3: 999}),
          (260000, [3, 4], {k: 500 + k % 97 for k in range(11, 260000, 613)})]


@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_wide_rows(shape, dtype):
    eng = E.gpu_engine(0)
    vt, xt = DT[dtype]
    n, short, long_rows = SHAPES[shape]
    rng = np.random.default_rng(shape)
    ln = np.resize(short, n)
    for r, k in long_rows.items():
        ln[r] = k
    pntr = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    # distinct ascending columns: a run from a random start, stretched where the row leaves room
    start, step = rng.integers(0, n, n), np.maximum(1, np.minimum(7, n // np.maximum(ln, 1)))
    start = np.minimum(start, n - np.maximum(ln * step, 1))
    at = np.arange(pntr[-1]) - np.repeat(pntr[:-1], ln)
    indx = (np.repeat(start, ln) + at * np.repeat(step, ln)).astype(np.int32)
    assert indx.min() >= 0 and indx.max() < n
    vals = rng.standard_normal(len(indx))
    p, i, v = (torch.tensor(a).cuda() for a in (pntr, indx, vals))
    v = v.to(vt)
    x = torch.tensor(rng.standard_normal((7, n))).to(xt).cuda()
    y0 = torch.tensor(rng.standard_normal((7, n))).to(xt).cuda()
    A = E.make_sparse_matrix(eng, n, p, i, v)
    B = E.make_sparse_matrix(eng, n, p, unaligned(i), unaligned(v))
    for mode in ("fused", "exact"):
        eng.set_spmv_mode(mode)
        for alpha, beta in ((1.0, 0.0), (-1.5, 0.0), (1.5, -2.0)):
            ref = y0.clone()
            for c in range(7):
                B.gemv("N", alpha, x[c], beta, ref[c])
            y = y0.clone()
            A.gemv("N", alpha, x[0], beta, y[0])
            assert torch.equal(y[0], ref[0]), (mode, alpha, beta)
            if dtype == "f64" and mode == "exact":
                assert np.array_equal(y[0].cpu().numpy(),
                                      O.spmv("N", n, n, alpha, pntr, indx, vals, x[0].cpu().numpy(), beta, y0[0].cpu().numpy()))
            if (alpha, beta) == (1.0, 0.0):
                y, d = torch.empty_like(y0[0]), torch.zeros(1, dtype=torch.float64, device="cuda")
                A.gemv_dot(x[0], y, d)
                parts = x[0].double() * y.double()
                assert torch.equal(y, ref[0])
                assert abs(d.item() - parts.sum().item()) <= n * torch.finfo(xt).eps * parts.abs().sum().item()
            for nrhs in (2, 3, 4, 5, 7):
                y = y0.clone()
                A.gemm(nrhs, alpha, x[:nrhs], beta, y[:nrhs])
                assert torch.equal(y[:nrhs], ref[:nrhs]) and torch.equal(y[nrhs:], y0[nrhs:]), (mode, alpha, beta, nrhs)

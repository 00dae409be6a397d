"""The staged product at the edges of its tiles: tiles of just under, exactly and just over the staged size, of the short
and of the long variant, empty rows, partial last tiles, and every split of several columns into passes.  In either mode
each column equals the product of the unstaged kernel (the route of arrays that are not 16-byte aligned) bit for bit;
in exact mode it equals the oracle's.  The transposed product is the oracle's bit for bit for every (alpha, beta)."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DT = {"f64": (torch.float64, torch.float64), "f32": (torch.float32, torch.float32), "bf16": (torch.bfloat16, torch.float32)}


def matrix(n, lengths, seed):
    rng = np.random.default_rng(seed)
    ln = np.minimum(np.resize(lengths, n), n)
    pntr = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    indx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in ln] + [np.zeros(0, int)]).astype(np.int32)
    return pntr, indx, rng.standard_normal(len(indx)), rng


def unaligned(t):
    """the same values at an address that is not a multiple of 16 bytes"""
    u = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:]
    u.copy_(t)
    assert u.data_ptr() % 16
    return u


# per 32 rows: 224 (one below is ragged), 255, 256, 257 entries; 240, 241 (the rule's line); 383, 384, 385; far above; none
SHAPES = [(1, [3]), (31, [7]), (33, [7, 6, 8]), (64, [8] * 31 + [7]), (96, [8]), (70, [8] * 31 + [9]), (100, [7, 8]),
          (101, [7] * 15 + [8] * 16 + [9]), (95, [12] * 31 + [11]), (160, [12]), (161, [12] * 31 + [13]), (300, [0, 5, 40]),
          (257, [0]), (1000, [0] * 31 + [200]), (9000, [7, 0, 12, 5])]


@pytest.mark.parametrize("dtype", ["f64", "f32", "bf16"])
@pytest.mark.parametrize("n,lengths", SHAPES)
def test_tiles(n, lengths, dtype):
    eng = E.gpu_engine(0)
    vt, xt = DT[dtype]
    pntr, indx, vals, rng = matrix(n, lengths, n)
    p, i, v = (torch.tensor(a).cuda() for a in (pntr, indx, vals))
    v = v.to(vt)
    x = torch.tensor(rng.standard_normal((11, n))).to(xt).cuda()
    y0 = torch.tensor(rng.standard_normal((11, n))).to(xt).cuda()
    A = E.make_sparse_matrix(eng, n, p, i, v)
    B = E.make_sparse_matrix(eng, n, p, unaligned(i) if len(indx) else i, unaligned(v) if len(indx) else v)
    for mode in ("fused", "exact"):
        eng.set_spmv_mode(mode)
        for alpha, beta in ((1.0, 0.0), (-1.5, 0.0), (1.0, 0.5), (1.5, -2.0)):
            ref = y0.clone()
            for c in range(11):
                B.gemv("N", alpha, x[c], beta, ref[c])
            y = y0.clone()
            A.gemv("N", alpha, x[0], beta, y[0])
            assert torch.equal(y[0], ref[0]), (mode, alpha, beta)
            if dtype == "f64" and mode == "exact":
                assert np.array_equal(y[0].cpu().numpy(),
                                      O.spmv("N", n, n, alpha, pntr, indx, vals, x[0].cpu().numpy(), beta, y0[0].cpu().numpy()))
            for nrhs in (1, 2, 3, 4, 5, 6, 7, 8, 11):
                y = y0.clone()
                A.gemm(nrhs, alpha, x[:nrhs], beta, y[:nrhs])
                assert torch.equal(y[:nrhs], ref[:nrhs]) and torch.equal(y[nrhs:], y0[nrhs:]), (mode, alpha, beta, nrhs)


@pytest.mark.parametrize("n,lengths", SHAPES)
def test_transposed(n, lengths):
    eng = E.gpu_engine(0)
    pntr, indx, vals, rng = matrix(n, lengths, n)
    x, y0 = rng.standard_normal(n), rng.standard_normal(n)
    A = E.make_sparse_matrix(eng, n, *(torch.tensor(a).cuda() for a in (pntr, indx, vals)))
    for alpha, beta in ((1.0, 0.0), (-1.5, 0.0), (1.0, 0.5), (1.5, -2.0)):
        y = torch.tensor(y0).cuda()
        A.gemv("T", alpha, torch.tensor(x).cuda(), beta, y)
        assert np.array_equal(y.cpu().numpy(), O.spmv("T", n, n, alpha, pntr, indx, vals, x, beta, y0)), (alpha, beta)

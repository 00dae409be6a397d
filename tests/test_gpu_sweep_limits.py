"""ILU(0) applications on patterns at the limits of the sweep plan (tests/test_sweep_plan.py plans them on the
host): bit for bit the oracle's, FP64 and FP32, 'N' and 'T'."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from oracle import oracle as O
from tests import test_sweep_plan as plan

pytestmark = pytest.mark.gpu
dev = torch.device("cuda")


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def values(pntr, indx, diag, rng):
    """off-diagonals in (-1, 1), diagonals above the row's sum"""
    v = rng.uniform(-1, 1, len(indx))
    v[diag] = 0.0
    rows = np.repeat(np.arange(len(diag)), np.diff(pntr))
    v[diag] = 1.0 + np.bincount(rows, weights=np.abs(v), minlength=len(diag))
    return v


@pytest.mark.parametrize("name", ["two_fields_260x260x16", "grid_70000x16x2", "grid_16384x16x3", "random_100000", "arrows_420_last"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_apply_bit_exact(eng, rng, name, dtype):
    p, i, d = plan.CASES[name]()
    n = len(p) - 1
    v = values(p, i, d, rng).astype(np.float64 if dtype == torch.float64 else np.float32)
    fo, do, _ = O.ilu_factor(p, i, v)
    ilu = E.make_ilu(eng, T(p), T(i), T(v))
    for k in range(2):      # the second round starts from what the first one left in the mailboxes
        x = rng.standard_normal(n).astype(v.dtype)
        assert np.array_equal(ilu.apply(T(x)).cpu().numpy(), O.ilu_apply(p, i, do, fo, x)), k
        assert np.array_equal(ilu.apply(T(x), trans="T").cpu().numpy(), O.ilu_apply(p, i, do, fo, x, trans="T")), k

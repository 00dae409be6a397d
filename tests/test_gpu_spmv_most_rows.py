"""Products of matrices with nearly 2^31 rows, whose last tiles end at the limit of a 32-bit row number; all rows but the last
70 are empty."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [2**31 - 40, 2**31 - 31, 2**31 - 1])
def test_last_rows(n, dtype):
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB")
    eng = E.gpu_engine(0)
    rng = np.random.default_rng(1)
    last = rng.integers(0, 9, 70)
    pntr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    pntr[-70:] = torch.tensor(np.cumsum(last).astype(np.int32)).cuda()
    indx = torch.tensor(np.concatenate([rng.permutation(16)[:k] for k in last]).astype(np.int32)).cuda()
    vals = torch.tensor(rng.integers(-8, 9, len(indx))).to(dtype).cuda()      # sums without rounding
    x = torch.tensor(rng.integers(-8, 9, 16)).to(dtype).cuda()
    y = torch.full((n,), float("nan"), dtype=dtype, device="cuda")
    E.sparse_gemv(eng, "N", n, 16, 1.0, pntr, indx, vals, x, 0.0, y)
    prod = (vals * x[indx.long()]).cpu().numpy()
    ends = np.cumsum(last)
    want = [prod[e - k:e].sum() for e, k in zip(ends, last)]
    assert y[-70:].tolist() == want
    for part in y[:-70].split(1 << 28):
        assert int(torch.count_nonzero(part)) == 0

"""The on-chip batch, whose inner products have FP32's exponent range, on matrices far from 1 and with inner tolerances whose
squares are below that range.  Every system has to meet its residual target, measured in FP64; a matrix scaled by
a power of two gives the unscaled one's solution scaled by it, bit for bit."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from hala_gb300 import problems as P

pytestmark = pytest.mark.gpu


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def batch(sizes, rng):
    sp, p, i, v = [0], [np.zeros(1, np.int64)], [], []
    for n in sizes:
        if n > 0:
            q, c, a = P.er_laplacian(n, rng)
        else:      # a diagonal system: the first inner iteration leaves no residual
            n = -n
            q, c, a = np.arange(n + 1), np.arange(n), np.full(n, 1.5)
        p.append(q[1:] + p[-1][-1])
        i.append(c + sp[-1])
        v.append(a)
        sp.append(sp[-1] + n)
    return (np.array(sp, np.int32), np.concatenate(p).astype(np.int32), np.concatenate(i).astype(np.int32),
            np.concatenate(v).astype(np.float32))


@pytest.mark.parametrize("power", [0, -118, -106, 100, 122])
@pytest.mark.parametrize("inner_rtol", [1e-4, 1e-21, 1e-30])
def test_range(eng, power, inner_rtol):
    rng = np.random.default_rng(5)
    sp, p, i, v = batch([1, -1, 40, -64, 300, 700, 1500, 3000], rng)
    b, x0 = rng.standard_normal(sp[-1]), rng.standard_normal(sp[-1])
    v2 = np.ldexp(v, power)      # exact: the entries lie in [0.01, 40]
    assert np.array_equal(np.ldexp(v2, -power), v)
    out = []
    for vals, scale in ((v, 1.0), (v2, 2.0 ** power)):
        B = E.gpu_batch(eng, T(sp), T(p), T(i), T(vals))
        x = T(x0 / scale)
        rel = torch.zeros(len(sp) - 1, dtype=torch.float64, device="cuda")
        B.solve(T(b), x, rtol=1e-11, inner_rtol=inner_rtol, relres=rel)
        assert np.all(rel.cpu().numpy() <= 1e-11)
        xs = x.cpu().numpy()
        r = b - P.csr_matvec(p, i, vals.astype(np.float64), xs)
        for s in range(len(sp) - 1):
            q = slice(sp[s], sp[s + 1])
            assert np.linalg.norm(r[q]) <= 1.01e-11 * np.linalg.norm(b[q]), s
        out.append(xs * scale)
    assert np.array_equal(out[0], out[1])

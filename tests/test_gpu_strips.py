"""The strip-scheduled triangular sweeps at the sizes where their plan changes: partly filled strips, strips
of unequal height, several strips per block, blocks in several thread-block clusters (mailboxes), rows
that blocks of two clusters read (watches), rows with more than three entries and more dependencies
than a block has slots (polled in memory).  FP64 and FP32 applications 'N' and 'T' are compared with
the oracle bit for bit."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from hala_gb300 import problems as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu
dev = torch.device("cuda")


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def stencil27(nx, ny, nz, rng):
    """the 27-point pattern, diagonally dominant random values"""
    offs = []
    for z in (-1, 0, 1):
        for y in (-1, 0, 1):
            for x in (-1, 0, 1):
                v = rng.uniform(-1, 1, nx * ny * nz) if (x, y, z) != (0, 0, 0) else np.full(nx * ny * nz, 27.0)
                offs.append(((x, y, z), v))
    return P._stencil_csr((nx, ny, nz), offs)


CASES = {
    "line_31": lambda rng: P.poisson2d(31, 1),
    "grid_33x17": lambda rng: P.poisson2d(33, 17),            # one strip, half a warp
    "grid_64x200": lambda rng: P.poisson2d(64, 200),          # strips of 32 lines, the last one short
    "grid_32x1200": lambda rng: P.poisson2d(32, 1200),        # more strips than a cluster of 16
    "grid_64x65x9": lambda rng: P.aniso3d(64, 65, 9),         # strips of 22, 22 and 21 lines
    "grid_32x33x70": lambda rng: P.aniso3d(32, 33, 70),       # many blocks: several clusters
    "grid_96x8x40": lambda rng: P.aniso3d(96, 8, 40),         # planes of fewer lines than a strip
    "grid_256x160x5": lambda rng: P.aniso3d(256, 160, 5),     # a plane over several blocks: two readers per row
    # odd grid lines: the factorisation's chunks end with the line
    "grid_63x65x61": lambda rng: P.aniso3d(63, 65, 61),
    "grid_301x97": lambda rng: P.poisson2d(301, 97),
    "stencil27_32x21x19": lambda rng: stencil27(32, 21, 19, rng),
    "random_30000": lambda rng: P.random_csr_sparse(30000, 12, rng),
}


@pytest.mark.parametrize("name", ["grid_33x17", "grid_64x65x9", "grid_301x97", "random_30000"])
def test_level_sets_of_chunked_factor(eng, rng, name):
    # the level sets come from the factorisation's chunks (lower) and from the level kernel's (upper)
    p, i, v = CASES[name](rng)
    do = O.diag_index(p, i)
    ilu = E.make_ilu(eng, T(p), T(i), T(v))
    for uplo in "LU":
        lev, nl = ilu.levels(uplo)
        lo, nlo = O.levels(p, i, do, uplo)
        assert nl == nlo and np.array_equal(lev.cpu().numpy(), lo)


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_strip_sweeps_bit_exact(eng, rng, name, dtype):
    p, i, v = CASES[name](rng)
    n = len(p) - 1
    v = v.astype(np.float64 if dtype == torch.float64 else np.float32)
    fo, do, _ = O.ilu_factor(p, i, v)
    ilu = E.make_ilu(eng, T(p), T(i), T(v))
    f, _ = ilu.factor()
    assert np.array_equal(f.cpu().numpy(), fo)
    for k in range(2):      # the second round starts from what the first one left in the mailboxes
        x = rng.standard_normal(n).astype(v.dtype)
        assert np.array_equal(ilu.apply(T(x)).cpu().numpy(), O.ilu_apply(p, i, do, fo, x)), k
        assert np.array_equal(ilu.apply(T(x), trans="T").cpu().numpy(), O.ilu_apply(p, i, do, fo, x, trans="T")), k

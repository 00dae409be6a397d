"""One GMRES cycle at the edges of its basis kernels: 8, 16 and 32 columns per group and one to each side, several
groups, rows that fill no warp, no CTA or exactly one.  The cycle's solution is the oracle's to 1e-9: rounding
(1e-16) times the operator's condition number (below 1e4) times the columns (at most 70) is 1e-10."""
import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from hala_gb300 import problems as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,restart", [(7, 1, 2), (51, 5, 8), (32, 8, 9), (257, 1, 7), (77, 13, 16), (77, 13, 17), (77, 13, 31), (77, 13, 32),
                                           (77, 13, 33), (241, 17, 1), (241, 17, 15), (241, 17, 40), (241, 17, 64), (241, 17, 65), (241, 17, 70)])
def test_one_cycle(nx, ny, restart):
    eng = E.gpu_engine(0)
    p, i, v = P.poisson2d(nx, ny)
    rng = np.random.default_rng(restart)
    b = rng.uniform(-1, 1, len(p) - 1)
    xo, ito = O.gmres(p, i, v, b, restart, max_iter=1)
    x = torch.zeros(len(b), dtype=torch.float64, device="cuda")
    gp, gi, gv, gb = (torch.tensor(a).cuda() for a in (p, i, v, b))
    it = E.solve_gmres(eng, E.stop_criteria(0.0, 1), restart, gp, gi, gv, gb, x)
    assert it == ito
    assert np.linalg.norm(x.cpu().numpy() - xo) <= 1e-9 * np.linalg.norm(xo)

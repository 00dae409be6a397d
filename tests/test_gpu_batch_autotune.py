"""Autotuning concerns the systems that do not fit on chip: a batch without any keeps its configuration, times nothing
and writes no cache line; the cache line of one with some is not taken for a batch with the same sizes and others streamed."""
import os

import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from hala_gb300 import problems as P

pytestmark = pytest.mark.gpu


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def star(n):
    """a hub coupled to every other row: 2 n - 2 + n entries, the hub's row too long to be kept on chip from n = 257"""
    A = np.eye(n) * 1.01
    A[0, 0] = 0.25 * (n - 1) + 0.01
    A[0, 1:] = A[1:, 0] = -0.25
    r, c = np.nonzero(A)
    return np.concatenate([[0], np.cumsum(np.bincount(r))]), c, A[r, c]


def batch(eng, systems):
    sp, p, i, v = [0], [np.zeros(1, np.int64)], [], []
    for q, c, a in systems:
        p.append(q[1:] + p[-1][-1])
        i.append(c + sp[-1])
        v.append(a)
        sp.append(sp[-1] + len(q) - 1)
    return sp[-1], E.gpu_batch(eng, T(np.array(sp, np.int32)), T(np.concatenate(p).astype(np.int32)),
                               T(np.concatenate(i).astype(np.int32)), T(np.concatenate(v).astype(np.float32)))


def lines(path):
    return open(path).read().splitlines() if os.path.exists(path) else []


def test_cache_lines(eng, tmp_path):
    rng = np.random.default_rng(3)
    cache = str(tmp_path / "tune.txt")
    er = [P.er_laplacian(n, rng) for n in (300, 300, 700)]
    n, onchip = batch(eng, er)
    b, x = T(rng.standard_normal(n)), torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    onchip.set_config(512, 64)
    assert onchip.autotune(b, x, 1e-8, cache) == (512, 64)
    assert lines(cache) == [] and torch.all(x == 7.0)
    for k, systems in enumerate(([star(300), er[1], er[2]], [er[0], er[1], star(700)]), 1):      # the same sizes, others streamed
        _, B = batch(eng, systems)
        best = B.autotune(b, x, 1e-8, cache)
        assert len(lines(cache)) == k and B.config == best
        assert B.autotune(b, x, 1e-8, cache) == best and len(lines(cache)) == k

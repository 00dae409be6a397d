"""Sweeps whose clusters start while the GPU is busy, so that a cluster's CTAs do not all begin at once: two
engines on streams of their own apply preconditioners of many blocks from two threads, beside short kernels on a
third stream.  Every application has the bits of the first one, made alone."""
import threading

import numpy as np
import pytest
import torch

from hala_gb300 import engine as E
from hala_gb300 import problems as P

pytestmark = pytest.mark.gpu
dev = torch.device("cuda")


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_busy_start(rng, dtype):
    jobs = []
    for shape in ((32, 33, 70), (64, 65, 9)):
        p, i, v = P.aniso3d(*shape)
        eng = E.gpu_engine(0)
        stream = torch.cuda.Stream()
        x = T(rng.standard_normal(len(p) - 1)).to(dtype)
        M = E.make_ilu(eng, T(p), T(i), T(v).to(dtype))
        alone = [M.apply(x, trans=t) for t in "NT"]
        torch.cuda.synchronize()
        eng.set_stream(stream)
        jobs.append((eng, stream, M, x, alone, []))

    def work(eng, stream, M, x, alone, wrong):
        with torch.cuda.stream(stream):
            for k in range(40):
                r = M.apply(x, trans="NT"[k & 1])
                if not torch.equal(r, alone[k & 1]):
                    wrong.append(k)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    side = torch.cuda.Stream()
    a = torch.ones(1 << 20, device=dev)
    with torch.cuda.stream(side):
        for _ in range(400):
            a.mul_(1.0)
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert [j[5] for j in jobs] == [[], []]

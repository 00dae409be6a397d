"""The host's plan of the triangular sweeps, checked without a GPU by tests/cpp/sweep_plan_check.cu: every packet
names its own row, all slots fit a CTA's shared memory, and a sweep over row numbers finds each entry where its
code says.  The patterns are at the plan's limits: grid lines longer than a strip and than 65,536 rows (a
packet's row offset has 16 bits), blocks with more rows of other blocks than slots, blocks whose own rows need
more slots than there are."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from hala_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "sweep_plan_check.cu")


def test_failing_allocations(tmp_path):
    """the planner's threads end, and the caller gets the exception, whichever allocation fails (a thread that cannot be
    started is done without)"""
    obj, exe = str(tmp_path / "check.o"), str(tmp_path / "alloc")
    inc = "-I" + os.path.join(ROOT, "include")
    for cmd in ([build.nvcc_path(), "-std=c++17", "-O2", *build.ARCH, inc, "-c", "-o", obj, SRC],
                [build.nvcc_path(), "-std=c++17", "-O2", "-o", exe, obj, os.path.join(os.path.dirname(SRC), "sweep_plan_alloc.cpp"), "-lpthread"]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("plan") / "sweep_plan_check.so")
    cmd = [build.nvcc_path(), "-std=c++17", "-O2", *build.ARCH, "-Xcompiler", "-fPIC", "-I" + os.path.join(ROOT, "include"), "-shared",
           "-o", out, SRC]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def by_distance(n, distances, keep=None):
    """(pntr, indx, diag) of the symmetric pattern with entries at the given distances; keep(d, rows): which rows i have i - d"""
    cols = np.concatenate([-np.array(sorted(distances, reverse=True)), [0], np.sort(distances)])
    rows = np.arange(n)
    ok = np.zeros((n, len(cols)), bool)
    for q, d in enumerate(cols):
        c = rows + d
        ok[:, q] = (c >= 0) & (c < n)
        if keep is not None and d != 0:
            hi = np.maximum(rows, c)
            ok[:, q] &= keep(abs(d), np.clip(hi, 0, n - 1))
    pntr = np.zeros(n + 1, np.int64)
    np.cumsum(ok.sum(1), out=pntr[1:])
    indx = (rows[:, None] + cols[None, :])[ok]
    diag = pntr[:-1] + ok[:, :len(distances)].sum(1)
    return pntr.astype(np.int32), indx.astype(np.int32), diag.astype(np.int32)


def grid(nx, ny, nz):
    return by_distance(nx * ny * nz, [1, nx, nx * ny],
                       lambda d, i: i % nx >= 1 if d == 1 else (i // nx % ny >= 1 if d == nx else i >= nx * ny))


def two_fields(nx, ny, nz):
    """two unknowns per grid point, one field after the other: each point's two unknowns are coupled"""
    m = nx * ny * nz
    return by_distance(2 * m, [1, nx, nx * ny, m],
                       lambda d, i: {1: i % nx >= 1, nx: i // nx % ny >= 1, nx * ny: i % m >= nx * ny, m: i >= m}[d])


def csr(A):
    A = (A + A.T + sp.eye(A.shape[0])).tocsr()
    A.sum_duplicates()
    A.sort_indices()
    rows = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), np.flatnonzero(rows == A.indices).astype(np.int32)


def random(n, degree):
    rng = np.random.default_rng(n + degree)
    m = n * degree // 2
    return csr(sp.coo_matrix((np.ones(m), (rng.integers(0, n, m), rng.integers(0, n, m))), shape=(n, n)))


def arrows(n, m, last):
    """blocks of m rows with a full first (or last) row and column"""
    i = np.arange(n)
    hub = np.minimum(i // m * m + (m - 1 if last else 0), n - 1)
    return csr(sp.coo_matrix((np.ones(n), (i, hub)), shape=(n, n)))


CASES = {
    "grid_33x17x5": lambda: grid(33, 17, 5),
    "grid_15x13x13": lambda: grid(15, 13, 13),
    "grid_64x65x30": lambda: grid(64, 65, 30),
    "grid_256x160x40": lambda: grid(256, 160, 40),
    "grid_16384x16x3": lambda: grid(16384, 16, 3),
    "grid_16385x16x3": lambda: grid(16385, 16, 3),
    "plane_of_65536": lambda: two_fields(256, 256, 16),
    "grid_70000x16x2": lambda: grid(70000, 16, 2),
    "two_fields_260x260x16": lambda: two_fields(260, 260, 16),
    "random_30000": lambda: random(30000, 12),
    "random_60000": lambda: random(60000, 6),
    "random_100000": lambda: random(100000, 12),
    "random_300000": lambda: random(300000, 3),
    "arrows_420_first": lambda: arrows(100800, 420, False),
    "arrows_420_last": lambda: arrows(100800, 420, True),
    "arrows_5": lambda: arrows(120000, 5, True),
}


@pytest.mark.parametrize("name", list(CASES))
def test_plan(lib, name):
    pntr, indx, diag = CASES[name]()
    n = len(pntr) - 1
    at = [a.ctypes.data_as(ctypes.c_void_p) for a in (pntr, indx, diag)]
    for xsize in (8, 4):
        for most in (16, 3):
            for nonunit_a, nonunit_b, rev_b in ((0, 1, 0), (1, 0, 1)):      # the applications of M and M^T
                bad, shape = (ctypes.c_long * 12)(), (ctypes.c_int * 8)()
                st = lib.sweep_plan_check(n, *at, xsize, most, nonunit_a, nonunit_b, rev_b, bad, shape)
                where = (name, xsize, most, rev_b, list(shape))
                assert st == 0, where
                found = np.array(list(bad)).reshape(2, 6)      # rows, slots, values, stuck steps, targets, strips
                assert not found.any(), (where, found.tolist())


def levels(pntr, indx, diag):
    lev = np.zeros(len(pntr) - 1, int)
    for r in range(len(lev)):
        for q in range(pntr[r], diag[r]):
            lev[r] = max(lev[r], lev[indx[q]] + 1)
    return int(lev.max()) + 1


def permuted(pattern, seed):
    pntr, indx, _ = pattern
    n = len(pntr) - 1
    q = np.random.default_rng(seed).permutation(n)
    return csr(sp.csr_matrix((np.ones(len(indx)), indx, pntr), shape=(n, n))[q][:, q])


# the most and the fewest steps of a sweep for each of the pattern's levels: strips of a grid in its order pipeline; in a random
# order, or where rows list more than three entries, they follow one another
PATHS = {
    "grid_63x65x61": (lambda: grid(63, 65, 61), 1.0, 2.0),
    "grid_15x13x13": (lambda: grid(15, 13, 13), 1.0, 1.6),      # planes of 13 lines: a strip each
    "grid_301x97": (lambda: grid(301, 97, 1), 1.0, 2.0),
    "line_5000": (lambda: grid(5000, 1, 1), 1.0, 1.1),
    "random_30000": (lambda: random(30000, 6), 50.0, 1e4),
    "grid_20x20x20_permuted": (lambda: permuted(grid(20, 20, 20), 1), 20.0, 1e4),
}


@pytest.mark.parametrize("name", list(PATHS))
def test_path(lib, name):
    make, fewest, most = PATHS[name]
    pntr, indx, diag = make()
    at = [a.ctypes.data_as(ctypes.c_void_p) for a in (pntr, indx, diag)]
    nlev = levels(pntr, indx, diag)
    for xsize in (8, 4):
        bad, shape = (ctypes.c_long * 12)(), (ctypes.c_int * 8)()
        assert lib.sweep_plan_check(len(pntr) - 1, *at, xsize, 16, 0, 1, 0, bad, shape) == 0
        for k in (0, 1):
            path, own = shape[4 * k + 2], shape[4 * k + 3]
            assert own <= nlev and fewest * nlev <= path <= most * nlev, (xsize, k, path, own, nlev)

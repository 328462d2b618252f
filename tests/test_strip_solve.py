"""Triangular solves and ILU(0) pipelined over strips of rows (strip_plan.h, strip_solve.cuh, strip_factor.cuh).

The plan is walked on the CPU with the kernel's rules, its actors in random order, and the walk's solution
is compared with the row recurrence's bit for bit (both round each product and sum as one fused operation).
On the GPU the solves are compared with the CPU recurrence in FP64 over sizes at the edges of steps, strips and
chunks: both subtract the same products in the same order, so the bar is the rounding of a few hundred thousand
chained operations of a diagonally dominant factor, 1e-13.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from fem_gb300 import lina, problems
from oracle import ilu as oilu
from oracle import port
from tests.conftest import ROOT, gpu_available


@pytest.fixture(scope="module")
def walker(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("strip") / "strip_plan.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fopenmp", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "fem_gb300", "csrc"), os.path.join(ROOT, "tests", "c", "strip_plan_driver.cpp"),
                    "-o", out], check=True)
    return C.CDLL(out)


def triangle(A, lower):
    """(ptr, col, val, 1/diagonal) of the strict triangle of A."""
    T = (sp.tril(A, -1) if lower else sp.triu(A, 1)).tocsr()
    T.sort_indices()
    return T.indptr.astype(np.int32), T.indices.astype(np.int32), T.data.copy(), 1.0 / A.diagonal()


def walk(lib, A, lower, b, seed=0):
    ptr, col, val, dinv = triangle(A, lower)
    x, info = np.full(len(b), np.nan), np.zeros(4, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rc = lib.strip_plan_walk(len(b), p(ptr), p(col), p(val), p(dinv), int(lower), p(b), p(x), C.c_uint(seed), p(info))
    return rc, x, info


def recurrence(A, lower, b):
    T = (sp.tril(A) if lower else sp.triu(A)).tocsr()
    return spla.spsolve_triangular(T, b, lower=lower)


def grid(m, k=None):
    """A nonsymmetric 7-point matrix on an m x k grid, diagonally dominant."""
    k = m if k is None else k
    n = m * k
    r, c = np.divmod(np.arange(n), k)
    rng = np.random.default_rng(m * 1000 + k)
    rows, cols = [], []
    for dr, dc in ((-1, -1), (-1, 0), (0, -1), (0, 1), (1, 0), (1, 1)):
        ok = (r + dr >= 0) & (r + dr < m) & (c + dc >= 0) & (c + dc < k)
        rows.append(np.nonzero(ok)[0])
        cols.append((r[ok] + dr) * k + c[ok] + dc)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    A = sp.coo_matrix((rng.uniform(-1, 1, len(rows)), (rows, cols)), shape=(n, n)) + sp.diags(4 + rng.random(n))
    A = A.tocsr()
    A.sort_indices()
    return A


def band(n, reach, per_row, seed):
    """Random symmetric pattern: per_row couplings of every row within reach."""
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), per_row)
    cols = np.clip(rows + rng.integers(-reach, reach + 1, len(rows)), 0, n - 1)
    A = sp.coo_matrix((rng.uniform(-1, 1, len(rows)), (rows, cols)), shape=(n, n))
    A = (A + A.T + sp.diags(4.0 * per_row + rng.random(n))).tocsr()
    A.sum_duplicates()
    A.sort_indices()
    return A


PATTERNS = {
    "one_row": lambda: grid(1),
    "short": lambda: grid(3),
    "one_strip": lambda: grid(30),
    "two_strips": lambda: grid(31),
    "strips": lambda: grid(97),
    "flat": lambda: grid(7, 500),
    "tall": lambda: grid(500, 7),
    "tridiagonal": lambda: grid(1, 700),
    "far": lambda: band(3000, 400, 1, 1),
    "long_rows": lambda: band(2000, 20, 5, 2),
    "elasticity": lambda: sp.csr_matrix((lambda s: (s.data, s.indices, s.indptr))(problems.elasticity_p1(9))),
}


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("name", PATTERNS)
def test_plan_walk_solves(walker, name, lower):
    A = PATTERNS[name]()
    b = np.random.default_rng(5).standard_normal(A.shape[0])
    ref = recurrence(A, lower, b)
    for seed in range(3):
        rc, x, info = walk(walker, A, lower, b, seed)
        assert rc in (0, 1), (rc, info)
        if rc == 0:
            assert np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max(), info
    if name in ("one_row", "short", "one_strip", "two_strips", "strips", "tridiagonal", "flat", "tall"):
        assert rc == 0


@pytest.mark.parametrize("lower", [True, False])
def test_wide_levels_get_no_plan(walker, lower):
    """Two levels of 1,000 and 9,000 rows, and a row of 17 entries in one triangle: other solves' work."""
    n, k = 10_000, 1_000
    rng = np.random.default_rng(12)
    rows = np.repeat(np.arange(k, n), 3)
    A = sp.coo_matrix((rng.uniform(-1, 1, len(rows)), (rows, rng.integers(0, k, len(rows)))), shape=(n, n))
    A = (A + A.T + sp.diags(10.0 + rng.random(n))).tocsr()
    A.sum_duplicates()
    A.sort_indices()
    assert walk(walker, A, lower, np.ones(n))[0] == 1
    D = sp.csr_matrix(np.ones((18, 18)) + 20 * np.eye(18))
    assert walk(walker, D, lower, np.ones(18))[0] == 1


@pytest.mark.parametrize("name", PATTERNS)
def test_factor_plan_walk_gives_the_factors(walker, name):
    A = PATTERNS[name]()
    ptr, col = A.indptr.astype(np.int32), A.indices.astype(np.int32)
    f, info = np.full(A.nnz, np.nan), np.zeros(4, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rc = walker.strip_factor_walk(A.shape[0], p(ptr), p(col), p(A.data), p(f), p(info))
    assert rc in (0, 1), (rc, info)
    if rc == 0:
        assert np.array_equal(f, oilu.ilu0(ptr, col, A.data)), info
    if name not in ("far", "long_rows", "elasticity"):
        assert rc == 0


def test_quotients_round_as_the_division(walker):
    walker.quotient_misses.restype = C.c_long
    assert walker.quotient_misses(C.c_long(5_000_000), C.c_uint(3)) == 0


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="no CUDA device")
@pytest.mark.parametrize("scale", [1.0, 1e-200, 1e-310])
@pytest.mark.parametrize("name", PATTERNS)
def test_gpu_factors_equal_restatement(name, scale):
    """Bit-identical factors, also where quotients leave the corrections' range (scaled rows) and are zeros."""
    A = PATTERNS[name]()
    data = A.data.copy()
    rows = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
    data[rows % 5 == 2] *= scale
    data[(rows + 1 == A.indices) & (rows % 7 == 3)] = 0.0
    ilu = lina.ILU(A.shape[0], A.indptr, A.indices, data)
    ref = port.ilu0(A.indptr, A.indices, data)
    assert np.array_equal(ilu.factor_values(), ref, equal_nan=True)
    ilu.refactor(2.0 * data)
    assert np.array_equal(ilu.factor_values(), port.ilu0(A.indptr, A.indices, 2.0 * data), equal_nan=True)


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="no CUDA device")
@pytest.mark.parametrize("name", PATTERNS)
def test_gpu_application_matches_recurrence(name):
    A = PATTERNS[name]()
    n = A.shape[0]
    ilu = lina.ILU(n, A.indptr, A.indices, A.data)
    F = sp.csr_matrix((ilu.factor_values(), A.indices, A.indptr), shape=(n, n))
    L, U = sp.tril(F, format="csr"), (sp.triu(F, 1) + sp.identity(n)).tocsr()
    r = np.random.default_rng(6).standard_normal(n)
    ref = spla.spsolve_triangular(U, spla.spsolve_triangular(L, r, lower=True), lower=False)
    z = ilu.apply(r)
    assert np.abs(z - ref).max() <= 1e-13 * np.abs(ref).max()
    z32 = ilu.apply(r, lina.PREC_MIXED)
    assert np.linalg.norm(z32 - ref) <= 1e-5 * np.linalg.norm(ref)
    for _ in range(3):
        assert np.array_equal(ilu.apply(r), z) and np.array_equal(ilu.apply(r, lina.PREC_MIXED), z32)


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="no CUDA device")
def test_gpu_application_passes_infinities_and_nans():
    """A right-hand side with an infinity and with NaNs (one of them with all bits set) ends, and gives NaN or
    infinity where the recurrence does."""
    A = grid(97)
    n = A.shape[0]
    ilu = lina.ILU(n, A.indptr, A.indices, A.data)
    F = sp.csr_matrix((ilu.factor_values(), A.indices, A.indptr), shape=(n, n))
    for at, v in ((n // 2, np.inf), (n // 3, np.nan), (40, np.array([-1], np.int64).view(np.float64)[0])):
        r = np.ones(n)
        r[at] = v
        bad = np.zeros(n, bool)
        bad[at] = True
        for T in (sp.tril(F, -1).tocsr(), sp.triu(F, 1).tocsr()):
            rows = range(n) if sp.triu(T).nnz == 0 else range(n - 1, -1, -1)
            for i in rows:
                bad[i] = bad[i] or bad[T.indices[T.indptr[i]:T.indptr[i + 1]]].any()
        for prec in (lina.PREC_FP64, lina.PREC_MIXED):
            z = ilu.apply(r, prec)
            assert np.array_equal(~np.isfinite(z), bad)

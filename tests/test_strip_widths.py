"""Strips of every width: rows of 1 to 4 entries held in registers and of up to 16 read where they are used, each with one
and with several strips, in the solves and (up to 4 on either side) in the factorisation.

The plan's walk on the CPU and the GPU solves are compared with the row recurrence exactly: all subtract the same
products in the same order, each as one fused operation, and multiply by the same 1 / diagonal.
"""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from fem_gb300 import lina
from oracle import ilu as oilu
from oracle import port
from tests.conftest import gpu_available
from tests.test_strip_rules import choice, rules  # noqa: F401
from tests.test_strip_solve import grid, triangle, walk, walker  # noqa: F401

gpu = pytest.mark.skipif(not gpu_available(), reason="no CUDA device")


def stencil(m, k, offsets):
    """A diagonally dominant matrix on an m x k grid with couplings to +-offsets."""
    n = m * k
    r, c = np.divmod(np.arange(n), k)
    rows, cols = [], []
    for dr, dc in offsets + [(-a, -b) for a, b in offsets]:
        ok = (r + dr >= 0) & (r + dr < m) & (c + dc >= 0) & (c + dc < k)
        rows.append(np.nonzero(ok)[0])
        cols.append((r[ok] + dr) * k + c[ok] + dc)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    rng = np.random.default_rng(m * 1000 + len(offsets))
    A = sp.coo_matrix((rng.uniform(-1, 1, len(rows)), (rows, cols)), shape=(n, n))
    A = (A + sp.diags(2.0 * len(offsets) + rng.random(n))).tocsr()
    A.sort_indices()
    return A


FIVE = [(0, 1), (1, 0)]
NINE = FIVE + [(1, 1), (1, -1)]
STAR = NINE + [(0, 2), (2, 0)]
WIDE = STAR + [(2, 1), (2, -1), (2, 2), (2, -2), (1, 2), (1, -2), (0, 3), (3, 0), (3, 1), (3, -1)]


def pair(m):
    return (sp.kron(grid(m), np.ones((2, 2))) + 20 * sp.identity(2 * m * m)).tocsr()


# name: matrix, entries per row (0: table), at least so many strips
WIDTHS = {
    "1_one": (lambda: grid(1, 700), 1, 1), "1_several": (lambda: stencil(400, 90, [(1, 0)]), 1, 2),
    "2_one": (lambda: stencil(29, 29, FIVE), 2, 1), "2_few": (lambda: stencil(31, 31, FIVE), 2, 2),
    "2_several": (lambda: stencil(97, 97, FIVE), 2, 4), "2_many": (lambda: stencil(200, 200, FIVE), 2, 7),
    "3_several": (lambda: grid(97), 3, 4),
    "4_one": (lambda: stencil(31, 31, NINE), 4, 1), "4_two": (lambda: stencil(97, 97, NINE), 4, 2),
    "4_several": (lambda: stencil(200, 200, NINE), 4, 4),
    "6_one": (lambda: stencil(40, 40, STAR), 0, 1), "6_several": (lambda: stencil(200, 200, STAR), 0, 4),
    "7_several": (lambda: pair(100), 0, 3), "16_one": (lambda: stencil(60, 60, WIDE), 0, 1),
    "16_two": (lambda: stencil(150, 150, WIDE), 0, 2),
}


def recurrence(lib, T, b, dt):
    """(ptr, col, val, dinv or None, lower), b: the fused row recurrence in dt."""
    ptr, col, val, dinv, lower = T
    f = lib.recurrence64 if dt == np.float64 else lib.recurrence32
    a = [ptr, col, val.astype(dt), None if dinv is None else dinv.astype(dt), b.astype(dt), np.zeros(len(b), dt)]
    p = lambda v: None if v is None else v.ctypes.data_as(C.c_void_p)  # noqa: E731
    f(len(b), p(a[0]), p(a[1]), p(a[2]), p(a[3]), int(lower), p(a[4]), p(a[5]))
    return a[5]


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("name", WIDTHS)
def test_walk_equals_the_recurrence(walker, rules, name, lower):  # noqa: F811
    make, width, strips = WIDTHS[name]
    A = make()
    b = np.random.default_rng(5).standard_normal(A.shape[0])
    used, out = choice(rules, A, lower)
    assert used == 3 and out[0] >= strips and out[1] == width
    ref = recurrence(rules, triangle(A, lower) + (lower,), b, np.float64)
    for seed in range(2):
        rc, x, info = walk(walker, A, lower, b, seed)
        assert rc == 0 and np.array_equal(x, ref), info


@pytest.mark.parametrize("name", [k for k in WIDTHS if WIDTHS[k][1]])
def test_factor_walk_gives_the_factors(walker, name):  # noqa: F811
    A = WIDTHS[name][0]()
    ptr, col = A.indptr.astype(np.int32), A.indices.astype(np.int32)
    f, info = np.full(A.nnz, np.nan), np.zeros(4, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert walker.strip_factor_walk(A.shape[0], p(ptr), p(col), p(A.data), p(f), p(info)) == 0, info
    assert info[1] == WIDTHS[name][1] and np.array_equal(f, oilu.ilu0(ptr, col, A.data))


@gpu
@pytest.mark.gpu
@pytest.mark.parametrize("name", WIDTHS)
def test_gpu_solves_equal_the_recurrence(rules, name):  # noqa: F811
    A = WIDTHS[name][0]()
    n = A.shape[0]
    ilu = lina.ILU(n, A.indptr, A.indices, A.data)
    f = port.ilu0(A.indptr, A.indices, A.data)
    assert np.array_equal(ilu.factor_values(), f)
    F = sp.csr_matrix((f, A.indices, A.indptr), shape=(n, n))
    L = triangle(F, True) + (True,)
    U = triangle(F, False)[:3] + (None, False)
    r = np.random.default_rng(8).standard_normal(n)
    for prec, dt in ((lina.PREC_FP64, np.float64), (lina.PREC_MIXED, np.float32)):
        ref = recurrence(rules, U, recurrence(rules, L, r, dt), dt)
        assert np.array_equal(ilu.apply(r, prec), ref.astype(np.float64))

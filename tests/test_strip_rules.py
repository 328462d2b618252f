"""Which triangular factors are solved over strips, and in which precision (strip::make_plan, strip::pays).

A chain of levels that each hold several steps of one strip takes the strips longer than the one-block solve; the
estimates that say so are host code, tested without a GPU against the times measured for such matrices.  On the GPU,
factors that take the strips in one precision only are applied like any other.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from fem_gb300 import lina
from oracle import port
from tests.conftest import ROOT, gpu_available
from tests.test_strip_solve import grid

gpu = pytest.mark.skipif(not gpu_available(), reason="no CUDA device")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("strip") / "strip_rules.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fopenmp", "-I" + os.path.join(ROOT, "fem_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c", "strip_rules_driver.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def choice(lib, A, lower):
    """(bits: 1 FP32, 2 FP64 on strips; -1 no plan), the driver's numbers."""
    T = (sp.tril(A, -1) if lower else sp.triu(A, 1)).tocsr()
    T.sort_indices()
    out = np.zeros(7)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    return lib.strip_rules(A.shape[0], p(T.indptr.astype(np.int32)), p(T.indices.astype(np.int32)), int(lower), p(out)), out


def lines(e, width, count, strips):
    """count lines of width points; a point couples to e points of the line before it, at the first line of each of the
    strips' equal shares to one.  Levels are lines: a strip walks ceil(width / 32) steps of each."""
    n = count * width
    r, c = np.divmod(np.arange(n), width)
    rows, cols = [], []
    for k in range(e):
        d = k - e // 2
        ok = (r > 0) & (c + d >= 0) & (c + d < width) & ((d == 0) | (r % (count // strips) != 0))
        rows.append(np.nonzero(ok)[0])
        cols.append((r[ok] - 1) * width + c[ok] + d)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    rng = np.random.default_rng(e * 1000 + width)
    A = sp.coo_matrix((rng.uniform(-1, 1, len(rows)), (rows, cols)), shape=(n, n))
    A = (A + A.T + sp.diags(2.0 * e + 2 + rng.random(n))).tocsr()
    A.sort_indices()
    return A


# entries, width, strips: the precisions that measured faster on strips (400 lines)
LINES = {(3, 60, 2): 3, (3, 120, 4): 1, (4, 120, 4): 1, (5, 60, 2): 3, (5, 120, 4): 0, (6, 120, 4): 0, (8, 60, 2): 3,
         (8, 120, 4): 1,
         (12, 60, 2): 1, (12, 120, 4): 0, (16, 60, 2): 3, (16, 120, 4): 1}


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("shape", LINES)
def test_several_steps_a_level_pay_where_they_measured_faster(rules, shape, lower):
    e, width, strips = shape
    got, out = choice(rules, lines(e, width, 400, strips), lower)
    assert got == LINES[shape], out


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("make", [lambda: grid(1), lambda: grid(31), lambda: grid(97), lambda: grid(200), lambda: grid(500, 7),
                                  lambda: grid(1, 700), lambda: sp.kron(grid(60), np.ones((2, 2))).tocsr()])
def test_mesh_matrices_keep_the_strips(rules, make, lower):
    got, out = choice(rules, make(), lower)
    assert got == 3, out


@gpu
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 120, 4), (12, 60, 2), (5, 120, 4), (16, 60, 2)])
def test_gpu_one_precision_on_strips(shape):
    """Strips in FP32 with one block in FP64, neither, and both: the recurrence's solution to rounding (as for all
    solves: 1e-13, in FP32 1e-5), the same bits each time, and bit-identical factors."""
    A = lines(shape[0], shape[1], 400, shape[2])
    n = A.shape[0]
    ilu = lina.ILU(n, A.indptr, A.indices, A.data)
    for scale in (1.0, 2.0):
        if scale != 1.0:
            ilu.refactor(scale * A.data)
        f = ilu.factor_values()
        assert np.array_equal(f, port.ilu0(A.indptr, A.indices, scale * A.data))
        F = sp.csr_matrix((f, A.indices, A.indptr), shape=(n, n))
        L, U = sp.tril(F, format="csr"), (sp.triu(F, 1) + sp.identity(n)).tocsr()
        r = np.random.default_rng(6).standard_normal(n)
        ref = spla.spsolve_triangular(U, spla.spsolve_triangular(L, r, lower=True), lower=False)
        z, z32 = ilu.apply(r), ilu.apply(r, lina.PREC_MIXED)
        assert np.abs(z - ref).max() <= 1e-13 * np.abs(ref).max()
        assert np.linalg.norm(z32 - ref) <= 1e-5 * np.linalg.norm(ref)
        assert np.array_equal(ilu.apply(r), z) and np.array_equal(ilu.apply(r, lina.PREC_MIXED), z32)


@gpu
@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda: grid(1, 700), lambda: grid(31), lambda: grid(97), lambda: grid(300),
                                  lambda: lines(3, 120, 400, 4),
                                  lambda: (sp.kron(grid(40), np.ones((2, 2))) + 20 * sp.identity(3200)).tocsr()])
def test_gpu_handles_without_memory_for_the_strips(make):
    """Where the strips' arrays do not fit, a handle takes the one-block solve and the row pool: same factors, same
    solutions, bit for bit, and less memory."""
    torch = pytest.importorskip("torch")
    A = make()
    n = A.shape[0]
    r = np.random.default_rng(6).standard_normal(n)
    out, held = [], []
    for limit in (0, 1):
        free = torch.cuda.mem_get_info()[0]
        lina.set_device_memory_limit(limit)
        try:
            ilu = lina.ILU(n, A.indptr, A.indices, A.data)
        finally:
            lina.set_device_memory_limit(0)
        held.append(free - torch.cuda.mem_get_info()[0])
        f = ilu.factor_values()
        ilu.refactor(0.5 * A.data)
        out.append([f, ilu.factor_values(), ilu.apply(r), ilu.apply(r, lina.PREC_MIXED)])
        ilu.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    if n >= 90000:
        assert held[1] < held[0]
    L, U = sp.tril(A, format="csr"), (sp.triu(A, 1) + sp.identity(n)).tocsr()
    z = []
    for limit in (0, 1):
        lina.set_device_memory_limit(limit)
        try:
            z.append(factors(L, U, r))
        finally:
            lina.set_device_memory_limit(0)
    assert np.array_equal(*z)


def factors(L, U, r):
    """U^-1 L^-1 r by a handle made from given factors."""
    h, p = C.c_void_p(), lambda a: a.ctypes.data_as(C.c_void_p)
    a = [np.ascontiguousarray(v) for T in (L, U) for v in (T.indptr.astype(np.int32), T.indices.astype(np.int32), T.data)]
    fn = lina.lib().lina_gpu_ilu_create
    fn.argtypes, fn.restype = [C.c_int] + [C.c_void_p] * 7, C.c_int
    assert fn(len(r), *[p(v) for v in a], C.addressof(h)) == 0, lina.last_error()
    x, z = lina.DeviceArray.from_host(r), lina.DeviceArray(len(r))
    assert lina.lib().lina_gpu_ilu_apply(h, lina.PREC_FP64, x.ptr, z.ptr) == 0
    out = z.to_host()
    lina.lib().lina_gpu_ilu_destroy(h)
    return out

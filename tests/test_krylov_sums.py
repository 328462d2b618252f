"""The Krylov kernels' reductions, the segmented batches' tasks and the FP32 V-cycle of long rows, at the sizes
where a task, a block or a rule of gpu_amg.cu ends."""
import numpy as np
import pytest
import scipy.sparse as sp

from fem_gb300 import lina, problems
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]


# tasks of 1,024 rows (systems of 49, 1,024, 1,089 and 4,225 rows), of 2,560 (1.4 million rows), and of 4,096 with a
# rest; the true residual may exceed the recurrence's by its rounding, for which the bar leaves as much again
@pytest.mark.parametrize("ms", [(7, 32, 33, 65), (840, 20, 839), (1603,)])
@pytest.mark.parametrize("prec", [lina.PREC_FP64, lina.PREC_MIXED])
def test_segmented_tasks(ms, prec):
    rng = np.random.default_rng(len(ms))
    systems = [problems.poisson_p1(m) for m in ms]
    bs = [rng.uniform(-1, 1, s.n) for s in systems]
    amgs = [lina.AMG.from_system(s, depth=problems.batch_depth(s.n), coarsening=lina.STANDARD, omega=0.6,
                                 smoother=lina.SMOOTHER_JACOBI, precision=prec) for s in systems]
    xs, infos = lina.SegmentedBatch(amgs).solve(bs, tol=1e-8, max_iter=300)
    for s, b, x, info in zip(systems, bs, xs, infos):
        assert info.status == 0
        A = sp.csr_matrix((s.data, s.indices, s.indptr), shape=(s.n, s.n))
        assert np.linalg.norm(b - A @ x) <= 2e-8 * np.linalg.norm(b)


# every sum and scalar of the iteration scales exactly with a right-hand side scaled by a power of two (nothing
# here comes near a subnormal number), so the iterates are the same numbers, scaled
@pytest.mark.parametrize("m", [9, 65, 257])
@pytest.mark.parametrize("history", [1, 2, 6])
def test_pcg_scales_exactly(m, history):
    s = problems.poisson_p1(m, seed=1)
    a = lina.AMG.from_system(s, depth=problems.batch_depth(s.n), coarsening=lina.STANDARD, smoother=lina.SMOOTHER_JACOBI, omega=0.6,
                             precision=lina.PREC_MIXED)
    a.set_fcg_history(history)
    x, info = a.pcg(s.b, tol=1e-8, max_iter=200)
    assert info.status == 0
    for e in (2.0 ** -50, 2.0 ** 50):
        xe, ie = a.pcg(s.b * e, tol=1e-8, max_iter=200)
        assert ie.iterations == info.iterations and np.array_equal(xe, x * e)


# the FP32 cycle against the FP64 cycle of the same hierarchy: unit roundoff 6e-8 times a condition number of the
# coarsest matrix of up to 1e4
@pytest.mark.parametrize("m", [97, 300, 513])
def test_fp32_cycle_of_long_rows(m):
    s = problems.elasticity_p1(m, degraded=False)
    r = np.random.default_rng(m).uniform(-1, 1, s.n)
    opts = dict(depth=problems.batch_depth(s.n), coarsening=lina.STANDARD, smoother=lina.SMOOTHER_JACOBI, omega=0.6)
    z32, z64 = (lina.AMG.from_system(s, precision=p, **opts).vcycle(r) for p in (lina.PREC_MIXED, lina.PREC_FP64))
    assert np.linalg.norm(z32 - z64) <= 6e-4 * np.linalg.norm(z64)


# a handle with a device-memory limit keeps the layouts without padding and the steps without images of their own;
# its sums run in another order: unit roundoff 1e-16 times about 100 products a row, ten passes and a condition
# number of the coarsest matrix of up to 1e3
@pytest.mark.parametrize("smoother", [lina.SMOOTHER_JACOBI, lina.SMOOTHER_MC_SOR])
def test_layouts_under_a_memory_limit(smoother):
    s = problems.elasticity_p1(150, degraded=False)
    r = np.random.default_rng(5).uniform(-1, 1, s.n)
    opts = dict(depth=problems.batch_depth(s.n), coarsening=lina.STANDARD, smoother=smoother, omega=0.6,
                precision=lina.PREC_FP64)
    free = lina.AMG.from_system(s, **opts)
    size = lina.lib().lina_gpu_amg_device_bytes(free.h)
    lina.set_device_memory_limit(size)
    try:
        lean = lina.AMG.from_system(s, **opts)
    finally:
        lina.set_device_memory_limit(0)
    assert lina.lib().lina_gpu_amg_device_bytes(lean.h) <= size
    z = free.vcycle(r)
    assert np.linalg.norm(lean.vcycle(r) - z) <= 1e-10 * np.linalg.norm(z)
    lean.update_values(2.0 * s.data)
    x, info = lean.pcg(s.b, tol=1e-8, max_iter=300)
    A = sp.csr_matrix((2.0 * s.data, s.indices, s.indptr), shape=(s.n, s.n))
    assert info.status == 0 and np.linalg.norm(s.b - A @ x) <= 2e-8 * np.linalg.norm(s.b)

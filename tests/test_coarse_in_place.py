"""A one-level hierarchy applied in place: the coarse solve reads all of its right-hand side while it writes the result,
so the library copies a vector that is both."""
import numpy as np
import pytest

from fem_gb300 import lina, problems
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]


@pytest.mark.parametrize("precision", [lina.PREC_FP64, lina.PREC_MIXED])
@pytest.mark.parametrize("m", [3, 9, 23])
def test_one_level_cycle_in_place(m, precision):
    s = problems.poisson_p1(m)
    a = lina.AMG.from_system(s, depth=1, coarsening=lina.STANDARD, smoother=lina.SMOOTHER_JACOBI, precision=precision)
    r = np.random.default_rng(m).uniform(-1, 1, s.n)
    z = a.vcycle(r)
    x = lina.DeviceArray.from_host(r)
    assert lina.lib().lina_gpu_vcycle(a.h, x.ptr, x.ptr) == 0
    assert np.isfinite(z).all() and np.array_equal(x.to_host(), z)

"""The bounded waits of the solves and the factorisation over strips (strip_solve.cuh: the helper lanes', the walking
warps' and the copying lane's) run out on entries that nothing publishes: every warp leaves, the copies it started have
landed, the error is reported, and the handle works on.
"""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from fem_gb300 import lina
from tests.conftest import gpu_available
from tests.test_strip_solve import grid

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

FACTORISATION = 2
LIMIT_US = 200000

# 7-point rows (entries in registers), and interleaved components (entries read where they are used)
MATRICES = {"registers": lambda: grid(97),
            "table": lambda: (sp.kron(grid(97), np.ones((2, 2))) + 20 * sp.identity(2 * 97 * 97)).tocsr()}


@pytest.mark.parametrize("what", [lina.PREC_FP64, lina.PREC_MIXED, FACTORISATION])
@pytest.mark.parametrize("name", MATRICES)
def test_waits_run_out(name, what):
    A = MATRICES[name]()
    ilu = lina.ILU(A.shape[0], A.indptr, A.indices, A.data)
    r = np.random.default_rng(2).standard_normal(A.shape[0])
    before = [ilu.factor_values(), ilu.apply(r), ilu.apply(r, lina.PREC_MIXED)]
    waited = C.c_double()
    rc = lina.lib().lina_gpu_ilu_wait_probe(ilu.h, what, LIMIT_US, C.byref(waited))
    if name == "table" and what == FACTORISATION:  # the row pool factorises it
        assert rc == lina.EINVAL
        return
    assert rc == lina.ECUDA and "ran out" in lina.last_error()
    assert LIMIT_US <= waited.value < LIMIT_US + 1.5e6
    after = [ilu.factor_values(), ilu.apply(r), ilu.apply(r, lina.PREC_MIXED)]
    assert all(np.array_equal(a, b) for a, b in zip(before, after))


def test_probe_arguments():
    A = grid(30)  # one strip: nothing to wait for
    ilu = lina.ILU(A.shape[0], A.indptr, A.indices, A.data)
    for what in (lina.PREC_FP64, lina.PREC_MIXED, FACTORISATION, 3):
        assert lina.lib().lina_gpu_ilu_wait_probe(ilu.h, what, LIMIT_US, None) == lina.EINVAL
    A = grid(97)
    ilu = lina.ILU(A.shape[0], A.indptr, A.indices, A.data)
    assert lina.lib().lina_gpu_ilu_wait_probe(ilu.h, lina.PREC_FP64, 0, None) == lina.EINVAL
    assert lina.lib().lina_gpu_ilu_wait_probe(ilu.h, 3, LIMIT_US, None) == lina.EINVAL

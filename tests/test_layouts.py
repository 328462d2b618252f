"""SpMV and damped Jacobi over the layouts and kernel variants the rules choose from (gpu_amg.cu), at the sizes
and row lengths where a variant, a batch of entries or a slice ends.

Bar: a row of k products summed in any order in a format of unit roundoff u is off by at most (k + 2) u |A| |x|,
and the sweep's update by a few u more of its own terms.
"""
import numpy as np
import pytest
import scipy.sparse as sp

from fem_gb300 import lina
from tests.conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]


def matrix(n, lengths, seed):
    """Rows of the given off-diagonal lengths (cycled) in a band, a dominant diagonal."""
    rng = np.random.default_rng(seed)
    ln = np.resize(np.asarray(lengths), n)
    rows = np.repeat(np.arange(n), ln)
    within = np.arange(len(rows)) - np.repeat(np.cumsum(ln) - ln, ln)
    cols = (rows + 1 + within * 3) % n
    A = sp.coo_matrix((rng.uniform(-1, 1, len(rows)), (rows, cols)), shape=(n, n)).tocsr()
    A = (A + sp.diags(2.0 + ln)).tocsr()
    A.sort_indices()
    return A


# entries per row: short rows (batches of eight and every rest), long rows, mixed; rows: one, a slice, the lane-group
# sizes, either side of one thread per row, and of the largest one-wave launch (155,648 rows)
CASES = [(1, [0]), (31, [0, 3]), (33, range(0, 18)), (700, range(0, 40)), (2049, [70, 3, 9]), (8001, range(1, 17)),
         (9000, [50, 60]), (32767, [6, 13]), (32768, [6, 13]), (32769, range(0, 24)), (40000, [40, 100]),
         (155648, [5, 6, 7]), (155649, [5, 6, 7]), (170001, [30])]


@pytest.mark.parametrize("quads", [1, 0])
@pytest.mark.parametrize("prec", [lina.PREC_FP64, lina.PREC_MIXED])
@pytest.mark.parametrize("n,lengths", CASES)
def test_products_and_sweeps(n, lengths, prec, quads):
    A = matrix(n, list(lengths), n)
    lina.set_sell_quads(quads)
    try:
        M = lina.Matrix(n, A.indptr, A.indices, A.data)
    finally:
        lina.set_sell_quads(1)
    u = 2.0 ** -24 if prec == lina.PREC_MIXED else 2.0 ** -53
    dt = np.float32 if prec == lina.PREC_MIXED else np.float64
    rng = np.random.default_rng(7)
    x, b = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, n).astype(dt)
    x64, b64 = x.astype(np.float64), b.astype(np.float64)
    S = abs(A) @ abs(x64)
    k = np.diff(A.indptr)
    assert (np.abs(M.spmv(x, prec) - A @ x64) <= (k + 4) * u * S).all()
    d = 1.0 / A.diagonal()
    ref = x64 + 0.6 * d * (b64 - A @ x64)
    bar = 0.6 * d * (k + 8) * u * (S + abs(b64)) + 4 * u * abs(x64)
    assert (np.abs(M.jacobi(b, x, 0.6, 1, prec) - ref) <= bar).all()

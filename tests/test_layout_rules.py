"""Which layout a matrix takes and which steps a level's layouts allow (layout_rules.h, gpu_amg.cu).

The rules are host code, tested without a GPU; on the GPU, levels at the edges of the rules give the same
V-cycles, bit for bit, whichever step they take.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from fem_gb300 import lina, problems
from tests.conftest import ROOT, gpu_available
from tests.test_layouts import matrix

gpu = pytest.mark.skipif(not gpu_available(), reason="no CUDA device")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rules") / "layout_rules.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "fem_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c", "layout_rules_driver.cpp"), "-o", out], check=True)
    lib = C.CDLL(out)
    lib.rule_lanes.argtypes = [C.c_long, C.c_int, C.c_void_p, C.c_long, C.c_int, C.c_long, C.c_int]
    lib.rule_lanes64.argtypes = [C.c_int, C.c_void_p, C.c_int]
    lib.rule_sell_variant.argtypes = [C.c_int, C.c_int, C.c_long]
    return lib


def pointers(n, lengths):
    """Row pointers of n rows whose lengths repeat."""
    return np.concatenate(([0], np.cumsum(np.resize(np.asarray(lengths, np.int64), n)))).astype(np.int32)


def lanes(rules, n, lengths, groups=0, lean=0, fused=24576, asked=0):
    ptr = pointers(n, lengths)
    return rules.rule_lanes(n, n, ptr.ctypes.data, groups, lean, fused, asked)


def test_fused_steps_need_lane_groups_everywhere(rules):
    """A three-coloured level of 33,000 rows of three entries: its colours keep lane groups where its natural-order
    matrix and its prolongation take one thread per row, so no fused step may read them in lane groups."""
    acol, a, p, r = lanes(rules, 33000, [3], 3), lanes(rules, 33000, [3]), lanes(rules, 33000, [1, 2]), lanes(rules, 11000, [3])
    assert acol > 0 and a == 0 and p == 0 and r > 0
    assert not rules.rule_fused(acol, a, r, p)
    for k in range(16):
        assert bool(rules.rule_fused(*[8 * (k >> i & 1) for i in range(4)])) == (k == 15)


def test_levels_within_the_row_limit_keep_lane_groups(rules):
    """Every level that lina_gpu_set_fused_rows admits is laid out for the fused step, up to 100,000 rows."""
    for limit in (24576, 32768, 33000, 49152, 99999):
        for n in (1000, 24576, 32767, 32768, 33000, 49152, 99999):
            if n <= limit:
                assert min(lanes(rules, n, [k], g, fused=limit) for k, g in ((3, 3), (14, 2), (3, 0), (60, 0))) > 0
        assert lanes(rules, limit + 1, [3], fused=limit) == 0
        assert lanes(rules, limit + 1, [14], fused=limit) == (0 if limit + 1 >= 32768 else 8)


def test_one_thread_per_row_only_where_it_is_no_slower(rules):
    """32,768 to 100,000 rows: even rows that fill the SMs take one thread per row; long rows among short ones, and row
    counts whose blocks divide badly among the SMs, keep the lane groups that measured faster."""
    for n, k in ((32768, 14), (33282, 14), (50748, 53), (66188, 53), (66049, 7), (75975, 95), (77000, 100), (99000, 5),
                 (31000, 5), (24577, 7)):
        assert lanes(rules, n, [k]) == 0, (n, k)
    for n, rows in ((24576, [5]), (31000, [8]), (36000, [250]), (45000, [200]), (80000, [100]), (90000, [60]), (90000, [200]),
                    (36000, [8] * 499 + [300]), (90000, [8] * 499 + [300]), (65000, [20] * 49 + [200]),
                    (90000, [4] * 4999 + [1500]), (45000, [60] * 49 + [250])):
        assert lanes(rules, n, rows) > 0, (n, rows[0])
    assert lanes(rules, 66000, [7], 4) == 0 and lanes(rules, 66000, [4] * 99 + [60], 4) > 0
    # at and above 100,000 rows, and in every asked-for layout, as before
    assert lanes(rules, 100000, [8] * 499 + [300]) == 0 and lanes(rules, 100000, [257]) == 8
    assert lanes(rules, 99999, [14], lean=1) == 8
    assert [lanes(rules, 50000, [14], asked=k) for k in range(1, 7)] == [0, 8, 4, 8, 16, 32]


def test_fp64_lanes_change_only_for_a_clear_gain(rules):
    """Other lanes than the layout's where they measured well under its time, the layout's where they measured over it."""
    def lanes64(n, rows, own):
        ptr = pointers(n, rows)
        return rules.rule_lanes64(n, ptr.ctypes.data, own)
    assert lanes64(18818, [14], 8) == 4 and lanes64(9214, [22], 8) == 4
    for n, k in ((24000, 100), (24000, 160), (32000, 130), (32000, 160), (32000, 200), (65000, 160), (9000, 80)):
        assert lanes64(n, [k], 8) == 8, (n, k)
    assert lanes64(90000, [4] * 9 + [16], 4) == 4 and lanes64(5000, [4] * 9 + [16], 4) == 4
    assert lanes64(2000, [4] * 999 + [700], 4) == 32
    for n in (0, 1, 31):
        assert lanes64(n, [1], 4) in (4, 8, 16, 32)


def test_layouts_asked_for_win(rules):
    """lina_gpu_set_layout(3..6) fixes the lanes of the staged colours as well, 1 keeps a batch's levels out of lane
    groups; 0 and 2 leave both to the rules."""
    few, many = np.array([300, 280, 4], np.int32), np.full(4000, 7, np.int32)
    stage = lambda v, n, asked: rules.rule_stage_lanes(v.ctypes.data_as(C.c_void_p), len(v), n, asked)  # noqa: E731
    for asked in (3, 4, 5, 6):
        assert stage(few, 4 << (asked - 3), asked) == stage(many, 4 << (asked - 3), asked) == 4 << (asked - 3)
    for asked in (0, 2):
        assert stage(few, 8, asked) == 32 and stage(many, 8, asked) == 1
    assert [rules.rule_groups_allowed(k) for k in range(7)] == [1, 0, 1, 1, 1, 1, 1]


def test_sell_variants_by_blocks_per_sm(rules):
    """Short, few, long, long with early loads (0 to 3), either side of one and four blocks of 256 rows an SM."""
    v = rules.rule_sell_variant
    assert [v(f64, 0, n) for f64 in (0, 1) for n in (32, 155648, 155680)] == [1, 1, 0, 1, 1, 0]
    assert [v(1, 1, n) for n in (32, 38944, 1 << 20)] == [3, 3, 3]
    assert [v(0, 1, n) for n in (32, 38912, 38944, 1 << 20)] == [3, 3, 2, 2]


def test_handles_with_a_memory_limit_hold_no_more(rules):
    """Their staged images are bounded by what images with 4-byte columns took (8 rows + 12 entries + 24 p bytes and the
    colours), their batches' tasks have 4,096 rows."""
    f = rules.rule_lean_images
    f.argtypes = [C.c_long] * 4
    size = lambda rows, c, p, e: 8 * rows + 12 * e + 24 * p + 4 * (c + 1 + 3)  # noqa: E731
    for c in (1, 4, 22):
        for rows, p in ((16, 1), (1600, 100), (9216, 576), (20000, 1252)):
            last = [e for e in range(0, 20000, 4) if f(rows, c, p, e)][-1]
            assert abs(size(rows, c, p, last) - 210 * 1024) <= 128
    # 9,216 rows of 14 entries over 16 blocks: 16-bit columns would fit, 4-byte columns do not
    assert f(9216, 12, 576, 9000) and not f(9216, 12, 576, 10752)
    assert [rules.rule_seg_chunk(n, lean) for n in (100, 608657, 5000000) for lean in (0, 1)] == [1024, 4096, 1024, 4096, 4096, 4096]


def ring(n):
    """Periodic second differences with a shift."""
    e = np.ones(n)
    A = sp.diags([2.1 * e, -e[:-1], -e[:-1], -1.0, -1.0], [0, 1, -1, n - 1, 1 - n], format="csr")
    A.sort_indices()
    return A


@gpu
@pytest.mark.gpu
@pytest.mark.parametrize("prec", [lina.PREC_FP64, lina.PREC_MIXED])
@pytest.mark.parametrize("n,lengths", [(155648, range(0, 18)), (155649, range(0, 18)), (38912, [23, 26, 40]),
                                       (38913, [23, 26, 40])])
def test_sell_variants_at_their_edges(n, lengths, prec):
    """Products and sweeps of the one-entry SELL layout either side of the variants' row counts.  Bar: k products summed
    in any order in a format of unit roundoff u are off by at most (k + 2) u |A| |x|, the update by a few u more."""
    A = matrix(n, list(lengths), n)
    lina.set_layout(1)
    lina.set_sell_quads(0)
    try:
        M = lina.Matrix(n, A.indptr, A.indices, A.data)
    finally:
        lina.set_layout(0)
        lina.set_sell_quads(1)
    u, dt = (2.0 ** -24, np.float32) if prec == lina.PREC_MIXED else (2.0 ** -53, np.float64)
    rng = np.random.default_rng(7)
    x, b = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, n).astype(dt)
    x64, b64 = x.astype(np.float64), b.astype(np.float64)
    S, k, d = abs(A) @ abs(x64), np.diff(A.indptr), 1.0 / A.diagonal()
    assert (np.abs(M.spmv(x, prec) - A @ x64) <= (k + 4) * u * S).all()
    ref = x64 + 0.6 * d * (b64 - A @ x64)
    assert (np.abs(M.jacobi(b, x, 0.6, 1, prec) - ref) <= 0.6 * d * (k + 8) * u * (S + abs(b64)) + 4 * u * abs(x64)).all()


@gpu
@pytest.mark.gpu
@pytest.mark.parametrize("precision", [lina.PREC_FP64, lina.PREC_MIXED])
def test_ring_level_above_32768_rows(precision):
    """An odd ring's inner level of about 33,300 rows and three colours with the largest documented row limit: in FP32
    its V-cycle step is fused (fewer launches), and V-cycles equal those of one launch per colour."""
    A = ring(66603)
    n = A.shape[0]
    r = np.random.default_rng(4).uniform(-1, 1, n)
    z, launches = [], []
    lina.set_sell_quads(0)  # one order of summation in the separate FP32 launches
    lina.set_fused_rows(49152)
    try:
        a = lina.AMG(n, A.indptr, A.indices, A.data, depth=4, coarsening=lina.STANDARD, smoother=lina.SMOOTHER_MC_SOR,
                     omega=1.0, precision=precision)
        for rows in (49152, lina.FUSED_ROWS_DEFAULT, 0):
            lina.set_fused_rows(rows)
            before = lina.launches()
            z.append(a.vcycle(r))
            launches.append(lina.launches() - before)
    finally:
        lina.set_fused_rows(lina.FUSED_ROWS_DEFAULT)
        lina.set_sell_quads(1)
    inner = len(a.sizes()) - 2
    assert a.level_size(inner) > 32768 and a.colours(inner).max() == 2
    assert np.isfinite(z[0]).all() and np.array_equal(z[0], z[1]) and np.array_equal(z[0], z[2])
    assert launches[1] < launches[2] and (launches[0] < launches[1]) == (precision == lina.PREC_MIXED)


@gpu
@pytest.mark.gpu
def test_one_thread_per_row_asked_for_in_a_batch():
    """Under lina_gpu_set_layout(1) a segmented batch has no lane groups, hence no fused steps: it issues the launches
    it issues with fused steps off, and solves alike."""
    systems = [problems.batch_system("elasticity" if i % 2 else "poisson", 600 + 100 * i, seed=i + 1) for i in range(4)]
    amgs = [lina.AMG.from_system(s, depth=1 + problems.batch_depth(s.n), coarsening=lina.STANDARD,
                                 smoother=lina.SMOOTHER_MC_SOR, omega=1.0, precision=lina.PREC_MIXED, matrix_tol=0.3)
            for s in systems]
    out = []
    for layout, rows in ((1, lina.FUSED_ROWS_DEFAULT), (1, 0), (0, lina.FUSED_ROWS_DEFAULT)):
        lina.set_layout(layout)
        lina.set_fused_rows(rows)
        try:
            batch = lina.SegmentedBatch(amgs)
            before = lina.launches()
            x, infos = batch.solve([s.b for s in systems], tol=1e-8, max_iter=1000, host_loop=True)
            out.append((x, [i.iterations for i in infos], lina.launches() - before))
        finally:
            lina.set_layout(0)
            lina.set_fused_rows(lina.FUSED_ROWS_DEFAULT)
    assert out[0][1] == out[1][1] and out[0][2] == out[1][2] > out[2][2]
    assert all(np.array_equal(a, b) for a, b in zip(out[0][0], out[1][0]))

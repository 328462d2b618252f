// layout_rules.h - host side of the storage layouts of a hierarchy's matrices: which layout a matrix takes, and
// which kernels its layouts allow.
#pragma once

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>
#include <vector>

namespace layout {

// Estimates of an FP64 sweep over a natural-order matrix, in cycles, for a group of S lanes per row (S = 1: one
// thread per row).  A sweep is bound by the SM's FP64 units (19 cycles a warp instruction and SM, whatever its
// active lanes: a warp's products are those of its longest row, then log2 S sums and two operations of the update)
// or by the chain of the longest row (1,180 cycles per batch of eight entries, or of four strides: two L2 round
// trips and the products).  Blocks of 256 threads do not divide evenly among 152 SMs: up to one and up to two blocks
// an SM cost as much as one and two, more cost about one block an SM more than their number (the scheduler fills
// some SMs further than others); for one thread per row, whose blocks are long, up to three cost 4.4.
struct Rows {
    long n = 0;
    double avg = 0.0;
    int longest = 0;
    double products[6] = {}, warps[6] = {};  // per log2 S: products of the warps' longest rows, warps
};

inline Rows row_counts(int n, const int* ptr) {
    Rows r;
    r.n = n;
    r.avg = n > 0 ? double(ptr[n] - ptr[0]) / n : 0.0;
    int longest = 0;
#pragma omp parallel for schedule(static) reduction(max : longest)
    for (int i = 0; i < n; i++) longest = std::max(longest, ptr[i + 1] - ptr[i]);
    r.longest = longest;
    for (int lg = 0; lg < 6; lg++) {
        if (lg == 1) continue;  // groups of two lanes are not used
        const int S = 1 << lg, per = 32 / S;
        const long warps = ((long)n + per - 1) / per;
        double products = 0.0;
#pragma omp parallel for schedule(static) reduction(+ : products)
        for (long w = 0; w < warps; w++) {
            int most = 0;
            for (long i = w * per; i < std::min<long>(n, (w + 1) * per); i++) most = std::max(most, ptr[i + 1] - ptr[i]);
            products += (most + S - 1) / S;
        }
        r.products[lg] = products;
        r.warps[lg] = double(warps);
    }
    return r;
}

inline double sweep_cycles(const Rows& r, int lg) {
    const int S = 1 << lg;
    const double blocks = std::max(1.0, std::ceil(double(r.n) * S / 256.0)), L = blocks / 152.0;
    const double full = L <= 1.0 ? 1.0 : L <= 2.0 ? 2.0 : lg == 0 && L < 3.0 ? 4.4 : L + 1.0;
    const double pipe = full / L * (r.products[lg] + r.warps[lg] * (lg + 2)) * 19.0 / 152.0;
    if (lg == 0) return 1500.0 + std::max(pipe, 1180.0 * ((r.longest + 7) / 8));
    const double chain = 0.6 * (1180.0 * ((r.longest + 4 * S - 1) / (4 * S)) + 90.0 * lg);
    // four lanes of long rows read half sectors of columns
    return (1500.0 + std::max(pipe, chain)) * (lg == 2 && r.avg > 64.0 ? 1.1 : 1.0);
}

// Lanes per row of the FP64 passes over a natural-order matrix whose layout has `lanes` (the arrays are the same for
// any number): those of the shortest estimate where it is under 0.85 of the layout's, for the estimates are good to
// about 15 %.  Measured over 355 shapes (600 to 99,000 rows of 4 to 300 entries, even and skewed) and the 96 levels
// of 17 hierarchies, GB300: on average 0.875 of the layout's lanes (the best choice: 0.86), 1.09 at worst (0.1 us);
// without the margin and with mean instead of counted products up to 1.32 (32,000 rows of 158 entries: 4 lanes
// 19.8 us, 8 lanes 15.0).  18,818 rows of 14 entries 4.8 (8 lanes) against 3.4 us (4), 13,011 of 94 8.8 (8)
// against 7.2 (16), 3,196 of 4 to 119 5.9 (4) against 3.7 (16).
inline int lanes64_for(const Rows& r, int lanes) {
    int best = 2, own = 2;
    for (int lg = 2; lg < 6; lg++) {
        if (sweep_cycles(r, lg) < sweep_cycles(r, best)) best = lg;
        if (1 << lg == lanes) own = lg;
    }
    return sweep_cycles(r, best) < 0.85 * sweep_cycles(r, own) ? 1 << best : lanes;
}

// Whether one thread per row suits a matrix of fewer than 100,000 rows (see lanes_for): not rows of more than
// 192 entries or much longer ones among short ones (a slice of 32 rows is padded to its longest, a thread walks it
// alone), nor, in natural order, where the estimate is longer than the lane groups'.  FP64 sweeps, one thread per
// row against lane groups (the layout chosen): 33,282 rows of 14 entries (3.2 us) against 4.3, 50,748 of 53 (9.5)
// against 10.0, 77,000 of 100 (16.8) against 23.5; 90,000 of 100 31.8 against (27.0), 45,000 of 200 29.2 against
// (23.6); 90,000 rows of 8 with 300 in every 500th 29.8 against (15.8), in FP32 without quads 16.4 against (8.7).
// lanes: the lane groups it would have otherwise.
inline bool one_thread_suits(const Rows& r, bool grouped, int lanes) {
    if (r.avg > 192.0 || r.longest > 3.0 * r.avg + 8.0) return false;
    if (grouped) return true;
    int lg = 2;
    while (1 << lg < lanes64_for(r, lanes)) lg++;
    return sweep_cycles(r, 0) <= 1.05 * sweep_cycles(r, lg);
}

// Layout choice, from sweeps of every level of elasticity (97 to 1,025 squared nodes) and Poisson hierarchies on
// GB300 in every layout.  One thread per row (SELL-32; long rows software-pipelined) from 100,000 rows on, and from
// 32,768 (rows of fewer than 8 entries: from 24,577, where 31,000 of 5 take 2.1 us against 4.4) where it suits the
// rows: there are enough of them, and each FP64 instruction does 32 rows' work (FP32 passes of such matrices read
// quads in either layout).  Below, a group of lanes per row, 8 lanes from 8k rows (enough rows to fill the GPU,
// several loads in flight per lane), wider groups below.  A colour-grouped matrix is swept colour by colour: its
// colours must have the rows to fill the GPU (groups: their number), or it 100,000 rows in all.
// n: the rows that the rule goes by (those of the largest system of a batch, or the matrix's).  lean: the lane
// groups' CSR arrays, which hold no padding, up to 100,000 rows (handles with a device-memory limit).  fused_rows:
// matrices of at most so many rows are read by fused steps, which need lane groups (0: none are).  asked: the
// layout of lina_gpu_set_layout.  Returns the lanes per row, 0 for one thread per row.
inline int lanes_for(long n, int rows, const int* ptr, long groups, bool lean, long fused_rows, int asked) {
    if (asked == 1) return 0;
    if (asked >= 3) return 4 << (asked - 3);
    const double avg = rows > 0 ? double(ptr[rows] - ptr[0]) / rows : 0.0;
    const int lanes = avg < 8.0 ? 4 : n >= 8000 ? 8 : avg >= 24.0 ? 16 : 8;
    if (asked != 0 || avg > 256.0) return lanes;
    if (n >= 100000) return 0;
    const bool many = groups > 0 ? avg < 24.0 && n >= 16384 * groups : n >= 32768 || (avg < 8.0 && n > 24576);
    if (lean || n <= fused_rows || !many) return lanes;
    return one_thread_suits(row_counts(rows, ptr), groups > 0, lanes) ? 0 : lanes;
}

// Variants of the one-thread-per-row kernel (sell_kernel) for a launch of npos rows.  SHORT rows in 32 registers, so
// that 64 warps an SM hide the latency; FEW of them with the rest of a row loaded together and the first entries
// before the wait for the previous kernel; LONG rows (mean of 24 and more) software-pipelined, with those first loads
// (EARLY) or without.  FEW pays up to a wave of its blocks, four an SM: repeated FP32 sweeps of 33,000 rows of 14
// entries 3.4 us SHORT, 2.0 FEW, of 155,000 3.9 and 2.9; a segmented batch 94 and 80 ms; a solve of 101,250 rows in
// FP64 5.83 and 5.30 ms, though repeated FP64 sweeps of such rows alone take 5.4 SHORT and 6.2 FEW.  (2.1M rows of 14
// in FP64: 82 us SHORT, 88 FEW.)  EARLY in FP32 takes registers: it wins up to a block an SM (33,000 rows of 30 4.3
// against 3.8 us, of 100 6.8 against 6.5; 50,000 of 100 7.4 against 8.5, 105,000 of 60 8.0 against 9.7), in FP64 it
// does not lose (33,000 of 30 5.4 against 4.9, 250,000 of 60 38 against 35).
enum SellVariant { SELL_SHORT = 0, SELL_FEW = 1, SELL_LONG = 2, SELL_LONG_EARLY = 3 };
constexpr long kBlockRows = 152L * 256;  // rows of one block on each SM
inline SellVariant sell_variant(bool f64, bool long_rows, long npos) {
    if (long_rows) return f64 || npos <= kBlockRows ? SELL_LONG_EARLY : SELL_LONG;
    return npos <= 4 * kBlockRows ? SELL_FEW : SELL_SHORT;
}

// A fused step reads all four matrices of a level as CSR, by groups of so many lanes: the colour-grouped and the
// natural-order copy of A, R and P follow rules of their own, so one of them can have lane groups (lanes > 0)
// where another, one thread per row, has neither lanes nor row pointers.
inline bool fused_layouts(int acol, int a, int r, int p) { return acol > 0 && a > 0 && r > 0 && p > 0; }

// A batch's staged steps lay their levels out in lane groups; a layout of one thread per row that was asked for wins.
inline bool groups_allowed(int asked) { return asked != 1; }

// FP64 lanes per row of a colour whose largest block's share has rows of these lengths (descending): the number
// with the shortest time, in cycles, of the longest warp (64 a product and 60 per batch of four, 115 a sum of the
// butterfly with its shuffles, 190 for the update) or of the SM's four FP64 units (64 an operation, shared by the
// block's warps).  lanes: the layout's, which a layout asked for with its lanes keeps.
inline int stage_lanes64(const std::vector<int>& len, int lanes, int asked) {
    if (asked >= 3) return lanes;
    int best = 4;
    long best_t = LONG_MAX;
    for (int S = 1, lg = 0; S <= 32; S *= 2, lg++) {
        const size_t per = 32 / S;
        long total = 0, longest = 0;
        for (size_t q = 0; q < len.size(); q += per) {
            const long products = (len[q] + S - 1) / S;
            total += products + lg + 2;
            longest = std::max(longest, 64 * products + 60 * ((products + 3) / 4) + 115 * lg + 190);
        }
        const long t = std::max(64 * ((total + 3) / 4), longest);
        if (t < best_t) {
            best = S;
            best_t = t;
        }
    }
    return best;
}

// Whether a handle with a device-memory limit has images for the staged steps of a level (of `rows` rows and c
// colours, the largest share of a block p rows and e entries): only where they would fit a block's 210 KB in FP64
// with columns of 4 bytes and no masks.  The images themselves are smaller, so such a handle holds no more for them
// than that size, and none for levels that only the smaller ones fit.
inline bool lean_images(size_t rows, size_t c, size_t p, size_t e) {
    auto pad = [](size_t v) { return (v + 3) / 4 * 4; };
    const size_t ints = pad(c + 1) + pad(p) + pad(p + 1) + pad(e), values = pad(e) + 2 * pad(p);
    return (rows * 8 + 15) / 16 * 16 + 8 * values + 4 * ints <= 210 * 1024;
}

// Rows per task of the segmented kernels: enough tasks for four blocks of 256 threads on each of the 152 SMs, of
// at least four rows a thread (a task's reduction costs as much as some rows) and at most 4,096.  16 systems of
// 608,657 rows in all, tasks of 1,024 rows with all loads of two or four rows in flight (before: 157 tasks of 4,096,
// a row at a time): r.z and z.q_j 16.2 us (28.9), p 11.9 (22.3), x and r 8.1 (18.6), p.q 4.8 (8.9).  Handles with a
// device-memory limit keep tasks of 4,096 rows, whose partials take a quarter of the memory.
inline int seg_chunk(int n, bool lean) {
    return lean ? 4096 : std::min(4096, std::max(1024, (n / (4 * 152) + 255) / 256 * 256));
}

}  // namespace layout

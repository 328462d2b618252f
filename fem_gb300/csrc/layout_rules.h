// layout_rules.h - host side of the storage layouts of a hierarchy's matrices: which layout a matrix takes, and
// which kernels its layouts allow.
#pragma once

#include <algorithm>
#include <climits>
#include <cstddef>
#include <vector>

namespace layout {

// Layout choice, from sweeps of every level of elasticity (97 to 1,025 squared nodes) and Poisson hierarchies on
// GB300 in every layout.  One thread per row (SELL-32; long rows software-pipelined) from 32,768 rows on: there
// are enough of them, and each FP64 instruction, which costs an SM 19 cycles whatever its active lanes, does 32
// rows' work (FP64 sweeps, one thread per row against 8 lanes per row: 34,814 rows of 8.5 entries 3.3 against
// 6.9 us, 50,748 rows of 53 entries 9.9 against 14.8, 70,011 of 95 19.7 against 24.0, 34,046 of 113 14.9 against
// 16.4; FP32 passes of such matrices read quads in either layout).  Below, a group of lanes per row, 8 lanes
// from 8k rows (enough rows to fill the GPU, several loads in flight per lane), wider groups below.  A
// colour-grouped matrix is swept colour by colour: its colours must have the rows to fill the GPU (groups: their
// number), or, as before, 100,000 rows in all.  lean: the lane groups' CSR arrays, which hold no padding, up to
// 100,000 rows (handles with a device-memory limit).  fused_rows: matrices of at most so many rows are read by fused
// steps, which need lane groups (0: none are).  asked: the layout of lina_gpu_set_layout.
// Returns the lanes per row, 0 for one thread per row.
inline int lanes_for_shape(long n, double avg, long groups, bool lean, long fused_rows, int asked) {
    if (asked == 1) return 0;
    if (asked >= 3) return 4 << (asked - 3);
    const bool many = n >= 100000 || (!lean && n > fused_rows &&
                                      (groups > 0 ? avg < 24.0 && n >= 16384 * groups : n >= 32768));
    if (asked == 0 && many && avg <= 256.0) return 0;
    if (avg < 8.0) return 4;
    if (n >= 8000) return 8;
    return avg >= 24.0 ? 16 : 8;
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

}  // namespace layout

// strip_plan.h - host side of the strip-pipelined triangular solves (strip_solve.cuh): which matrices suit
// them, and the layout of the strips' steps.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define STRIP_HD __host__ __device__
#else
#define STRIP_HD
#endif

namespace strip {

constexpr int kSteps = 8;                  // steps per chunk (one stage of shared memory)
constexpr int kPos = 32 * kSteps;          // positions per chunk
constexpr int kHelpers = 2;                // helper warps
constexpr int kThreads = 32 * (2 + kHelpers);
constexpr int kRingMin = 16, kRingMax = 64;  // steps a strip keeps in shared memory: more than a chunk
constexpr int kSlots = 512;                // hand-over slots: the fetched entries of two chunks fit
constexpr int kMaxStrips = 148;            // one block per SM, a few left free
constexpr int kRowsPerStrip = 30;          // rows of the widest level per strip: a step holds 32
constexpr int kMaxEntries = 16;            // entries of a row (stage size)
constexpr int kSmemMax = 200 * 1024;
constexpr int kLag = 25;                   // steps an exchange between strips takes, about (2 us, in FP32)

// The plan of one factor: positions are chunk * 256 + step * 32 + lane.
struct Plan {
    int strips = 0;      // 0: the matrix does not suit the strips
    int chunks = 0;
    int ring = 0;        // steps kept (a power of two)
    int width = 0;       // entries per row of every chunk where that is at most 4, else 0 (table)
    int max_width = 0;
    double ns32 = 0.0, ns64 = 0.0;     // estimated time of a solve in FP32, in FP64
    double win32 = 0.0, win64 = 0.0;   // and of the one-block solve of the same levels
    std::vector<int> first;            // first chunk of each strip (strips + 1)
    std::vector<int> ext_first;        // first fetched entry of each strip (strips + 1)
    std::vector<int> ext;              // row of each fetched entry
    std::vector<int> table;            // per chunk: offset of its entries, entries per row, end of its fetched entries, 0
    std::vector<int> row;              // row of each position, -1 none
    std::vector<int> enc, perm;        // per entry: the place of its operand in shared memory; its value's index
    long entries() const { return (long)enc.size(); }
    size_t positions() const { return (size_t)chunks * kPos; }
};

// Times on GB300 in ns.  A step of w entries a row, held in registers (fixed: every row has w <= 4 of them) or read where
// they are used (in groups of four and singly): from chains of 20,000 and 400 levels of 16 rows.  A level of the
// one-block solve whose rows have up to e entries: the same chains (levels of more rows take longer; so an estimate
// below it is a gain; only rows of mostly 8 or 16 entries are counted longer, whose entries lie a multiple of the banks
// apart: 128 rows of 8 take 0.19 us a level more, of 16 0.8).  An exchange between strips takes 2.4 us.
constexpr double kLagNs = 2400.0;
inline double step_ns(int w, bool fixed, bool f64) {
    if (fixed) return f64 ? 76.0 + 43.0 * w : 62.0 + 4.5 * w;
    return f64 ? 110.0 + 197.0 * (w / 4) + 58.0 * (w % 4) : 110.0 + 40.0 * (w / 4) + 55.0 * (w % 4);
}
inline double level_ns(int e, bool f64) {
    constexpr double t32[kMaxEntries + 1] = {540, 550, 580, 580, 655, 680, 684, 715, 752,
                                             752, 753, 754, 755, 780, 820, 850, 879};
    constexpr double t64[kMaxEntries + 1] = {600,  606,  685,  685,  861,  879,  881,  1040, 1216,
                                             1217, 1218, 1219, 1220, 1220, 1220, 1220, 1930};
    return f64 ? t64[e] : t32[e];
}
inline double conflict_ns(int e, int rows, long entries) {
    return (e == 8 || e == 16) && entries >= 0.9 * e * rows ? (e == 8 ? 0.12 : 0.33) * entries : 0.0;
}

// Rows listed level by level (order, with lev[i] the level of row i, nlev levels), row i's entries
// [beg_i, end_i) of col.  lower: a row needs smaller indices.  Returns false (no plan) where
//  - the widest level has more than 4,440 rows: the levels are wide enough for the other solves;
//  - a row has more than 16 entries (stages of shared memory);
//  - more than 8 entries per step come from other strips, which the helper warps could not fetch in
//    the time of a step (64 lanes, an L2 round trip each);
//  - a chunk has more than 256 fetched entries (it and the next one share the slots);
//  - the pipeline, followed step by step with an exchange of kLag steps, takes more than 4 steps per level.
// Whether it is faster than the one-block solve, where there is one, its estimates say (pays).
inline bool make_plan(Plan& P, int n, const std::vector<int>& order, const std::vector<int>& lev, int nlev,
                      const std::vector<int>& beg, const std::vector<int>& end, const int* col, bool lower) {
    P = Plan();
    if (n <= 0 || nlev <= 0) return false;
    std::vector<int> width(nlev, 0);
    int maxw = 0, maxe = 1;
    for (int i = 0; i < n; i++) {
        maxw = std::max(maxw, ++width[lev[i]]);
        maxe = std::max(maxe, end[i] - beg[i]);
    }
    if (maxw > kMaxStrips * kRowsPerStrip || maxe > kMaxEntries) return false;
    const int K = std::max(1, std::min(n, (maxw + kRowsPerStrip - 1) / kRowsPerStrip));
    auto strip_of = [&](int i) { return (int)((long)(lower ? i : n - 1 - i) * K / n); };
    // rows by strip, then level
    std::vector<int> start(K + 1, 0), rows(n), stepof(n);
    for (int i = 0; i < n; i++) start[strip_of(i) + 1]++;
    for (int s = 0; s < K; s++) start[s + 1] += start[s];
    {
        std::vector<int> at(start.begin(), start.end() - 1);
        for (int t = 0; t < n; t++) rows[at[strip_of(order[t])]++] = order[t];
    }
    // steps: up to 32 rows of one level; stepof = step within the strip * 32 + lane
    std::vector<int> nsteps(K, 0);
#pragma omp parallel for schedule(dynamic, 1)
    for (int s = 0; s < K; s++) {
        int step = -1, lane = 32, level = -1;
        for (int t = start[s]; t < start[s + 1]; t++) {
            const int i = rows[t];
            if (lane == 32 || lev[i] != level) {
                step++;
                lane = 0;
                level = lev[i];
            }
            stepof[i] = step * 32 + lane++;
        }
        nsteps[s] = step + 1;
    }
    // how far back a strip's rows reach within it
    int look = 1;
#pragma omp parallel for schedule(static) reduction(max : look)
    for (int i = 0; i < n; i++)
        for (int p = beg[i]; p < end[i]; p++)
            if (strip_of(col[p]) == strip_of(i)) look = std::max(look, stepof[i] / 32 - stepof[col[p]] / 32);
    P.ring = kRingMin;
    while (P.ring < look + 1 && P.ring < kRingMax) P.ring *= 2;
    const int ring = P.ring;
    auto fetched = [&](int i, int j) {
        return strip_of(i) != strip_of(j) || stepof[i] / 32 - stepof[j] / 32 >= ring;
    };
    P.first.assign(K + 1, 0);
    for (int s = 0; s < K; s++) P.first[s + 1] = P.first[s] + (nsteps[s] + kSteps - 1) / kSteps;
    P.chunks = P.first[K];
    P.max_width = maxe;
    P.width = maxe <= 4 ? maxe : 0;
    // entries per row of every chunk
    P.table.assign(4 * (size_t)P.chunks, 0);
#pragma omp parallel for schedule(dynamic, 1)
    for (int s = 0; s < K; s++)
        for (int t = start[s]; t < start[s + 1]; t++) {
            int& w = P.table[4 * (size_t)(P.first[s] + stepof[rows[t]] / kPos) + 1];
            w = P.width ? P.width : std::max(w, end[rows[t]] - beg[rows[t]]);
        }
    long total = 0, steps = 0;
    for (int c = 0; c < P.chunks; c++) {
        P.table[4 * (size_t)c] = (int)total;
        total += (long)P.table[4 * (size_t)c + 1] * kPos;
        if (total > INT32_MAX / 2) return false;
    }
    for (int s = 0; s < K; s++) steps += nsteps[s];
    if (P.positions() > (size_t)INT32_MAX / 2) return false;
    const int empty = ring * 32 + kSlots;  // a word that holds zero, for padding
    P.row.assign(P.positions(), -1);
    P.enc.assign(total, empty);
    P.perm.assign(total, -1);
    std::vector<std::vector<int>> ext(K), ext_step(K);
#pragma omp parallel for schedule(dynamic, 1)
    for (int s = 0; s < K; s++) {
        int t = start[s];
        std::vector<int>& x = ext[s];
        for (int step = 0; step < nsteps[s]; step++) {
            int t1 = t;
            while (t1 < start[s + 1] && stepof[rows[t1]] / 32 == step) t1++;
            const int c = P.first[s] + step / kSteps;
            const size_t at = (size_t)P.table[4 * (size_t)c] + 32 * (size_t)(step % kSteps);
            for (int u = t; u < t1; u++) P.row[(size_t)c * kPos + 32 * (size_t)(step % kSteps) + (u - t)] = rows[u];
            for (int k = 0; k < P.table[4 * (size_t)c + 1]; k++)  // fetched entries are numbered entry by entry
                for (int u = t; u < t1; u++) {
                    const int i = rows[u], p = beg[i] + k;
                    if (p >= end[i]) continue;
                    const size_t q = at + (size_t)k * kPos + (u - t);
                    P.perm[q] = p;
                    if (fetched(i, col[p])) {
                        P.enc[q] = ring * 32 + (int)(x.size() % kSlots);
                        x.push_back(col[p]);
                        ext_step[s].push_back(step);
                    } else {
                        P.enc[q] = (stepof[col[p]] / 32 % ring) * 32 + stepof[col[p]] % 32;
                    }
                }
            t = t1;
            P.table[4 * (size_t)c + 2] = (int)x.size();
        }
    }
    for (int s = 0; s < K; s++)
        for (int c = P.first[s]; c < P.first[s + 1]; c++)
            if (P.table[4 * (size_t)c + 2] - (c == P.first[s] ? 0 : P.table[4 * (size_t)c - 2]) > kSlots / 2) return false;
    P.ext_first.assign(K + 1, 0);
    for (int s = 0; s < K; s++) P.ext_first[s + 1] = P.ext_first[s] + (int)ext[s].size();
    P.ext.resize(P.ext_first[K]);
    for (int s = 0; s < K; s++) std::copy(ext[s].begin(), ext[s].end(), P.ext.begin() + P.ext_first[s]);
    if ((long)P.ext.size() > 8 * steps) return false;
    // the pipeline in units of a step, and in ns: a step starts when the one before it and its chunk's fetched entries
    // are there
    struct Time {
        double v[3];
    };
    std::vector<std::vector<Time>> done(K);
    Time last = {};
    const double lag[3] = {kLag, kLagNs, kLagNs};
    for (int s = 0; s < K; s++) {
        done[s].assign(nsteps[s], Time{});
        size_t e = 0;
        Time now = {};
        for (int step = 0; step < nsteps[s]; step++) {
            for (; e < ext[s].size() && ext_step[s][e] / kSteps == step / kSteps; e++) {
                const int j = ext[s][e];
                for (int k = 0; k < 3; k++) now.v[k] = std::max(now.v[k], done[strip_of(j)][stepof[j] / 32].v[k] + lag[k]);
            }
            const int w = P.table[4 * (size_t)(P.first[s] + step / kSteps) + 1];
            now.v[0] += 1.0;
            now.v[1] += step_ns(w, P.width > 0, false);
            now.v[2] += step_ns(w, P.width > 0, true);
            done[s][step] = now;
        }
        for (int k = 0; k < 3; k++) last.v[k] = std::max(last.v[k], now.v[k]);
    }
    if (last.v[0] > 4.0 * nlev + 4.0 * kLag) return false;
    P.ns32 = last.v[1];
    P.ns64 = last.v[2];
    std::vector<int> most(nlev, 0);
    std::vector<long> entries(nlev, 0);
    for (int i = 0; i < n; i++) {
        most[lev[i]] = std::max(most[lev[i]], end[i] - beg[i]);
        entries[lev[i]] += end[i] - beg[i];
    }
    for (int l = 0; l < nlev; l++) {
        P.win32 += level_ns(most[l], false) + conflict_ns(most[l], width[l], entries[l]);
        P.win64 += level_ns(most[l], true) + conflict_ns(most[l], width[l], entries[l]);
    }
    P.strips = K;
    return true;
}

// Whether the strips are used where the one-block solve is there too.  Most mesh matrices gain 1.4 to 5 times in either
// precision (5- to 13-point grids, Delaunay meshes, interleaved components).  Few do not: levels that cross few
// strips, so that a strip walks several steps of each (four strips of 100 lines of 120 points, coupled to the
// line before by e points: FP64 569 us one block, 656 strips for e = 3, 722 and 1,163 for 5, 1,003 and 2,174 for
// 12; FP32 478 and 228, 557 and 677, 685 and 776).
inline bool pays(const Plan& P, bool f64) { return f64 ? P.ns64 <= P.win64 : P.ns32 <= P.win32; }

// ---------------------------------------------------------------- the ILU(0) factorisation on the strips
// A row of the factorisation needs the upper entries U_kj of the rows k its lower entries name: the
// dependencies of the lower solve, so its steps are walked.  A row's entries are held as W lower ones (as
// many padding ones first as it has fewer), the diagonal and W upper ones; a "pair" is a product
// L_ik U_kj of a lower entry k (slot q) in the sum of a later entry j (a lower slot > q, the diagonal, an
// upper slot).  The pairs are numbered by entry, then by q, the order in which the sums take them.
constexpr int kFactorWidth = 4;
STRIP_HD constexpr int pairs_of(int W) { return W * (W - 1) / 2 + W + W * W; }
STRIP_HD constexpr int pair_index(int W, int entry, int q) {  // entry: lower slot, W the diagonal, W + 1 + t an upper slot
    return entry < W ? entry * (entry - 1) / 2 + q : W * (W - 1) / 2 + (entry - W) * W + q;
}

// Quotients a / d of one row share the reciprocal of d.  Markstein's method ("Computation of elementary functions
// on the IBM RISC System/6000 processor", 1990): with r = 1 / d rounded to nearest, a q within a few ulps of
// a / d is corrected by its exact remainder, q + (a - d q) r; the second correction rounds as the quotient
// does.  Only for exponents within +-400 of 0 (or a = 0, where a r has the right sign), so that no remainder
// loses bits; exponents are looked at as integers.
STRIP_HD inline bool mid_range(unsigned high_word) {
    const unsigned e = (high_word >> 20) & 0x7ffu;
    return e >= 1023u - 400u && e <= 1023u + 400u;
}

struct FactorPlan {
    int width = 0;                // 0: none
    unsigned used = 0;            // pairs that some row has
    std::vector<int> rec;         // per position: first entry of the row in CSR, lower entries | upper entries << 8
    std::vector<short> place;     // per chunk and pair: where U_kj is in shared memory, -1 none
    std::vector<int> ext_first, ext;  // fetched entries: the CSR entry of U_kj
    std::vector<int> ext_end;     // per chunk: end of its fetched entries within its strip's
};

// On the lower factor's plan.  False where a row has more than four entries on either side of the diagonal or
// none on it, or where the fetched entries of a chunk exceed the slots.
inline bool make_factor_plan(FactorPlan& F, const Plan& P, int n, const int* ptr, const int* col,
                             const std::vector<int>& diag) {
    F = FactorPlan();
    if (!P.strips || !P.width) return false;
    int W = 1, bad = 0;
#pragma omp parallel for schedule(static) reduction(max : W) reduction(| : bad)
    for (int i = 0; i < n; i++) {
        if (diag[i] < 0) bad = 1;
        W = std::max(W, std::max(diag[i] - ptr[i], ptr[i + 1] - 1 - diag[i]));
    }
    if (bad || W > kFactorWidth) return false;
    const int NP = pairs_of(W), rw = P.ring * 32;
    std::vector<int> pos(n);  // chunk * 256 + step * 32 + lane
#pragma omp parallel for schedule(static)
    for (size_t t = 0; t < P.positions(); t++)
        if (P.row[t] >= 0) pos[P.row[t]] = (int)t;
    F.rec.assign(2 * P.positions(), 0);
    for (size_t t = 0; t < P.positions(); t++)
        if (P.row[t] < 0) F.rec[2 * t] = -1;
    F.place.assign(P.positions() * NP, -1);
    F.ext_end.assign(P.chunks, 0);
    F.ext_first.assign(P.strips + 1, 0);
    std::vector<std::vector<int>> ext(P.strips);
    unsigned used = 0;
#pragma omp parallel for schedule(dynamic, 1) reduction(| : used, bad)
    for (int s = 0; s < P.strips; s++) {
        std::vector<int>& x = ext[s];
        const int lo = P.first[s] * kPos, hi = P.first[s + 1] * kPos;
        for (int c = P.first[s]; c < P.first[s + 1]; c++) {
            const size_t before = x.size();
            for (int st = 0; st < kSteps; st++) {
                int src[pairs_of(kFactorWidth)][32];  // per pair and lane: the CSR entry of U_kj
                for (int k = 0; k < NP; k++)
                    for (int l = 0; l < 32; l++) src[k][l] = -1;
                const size_t p0 = (size_t)c * kPos + 32 * (size_t)st;
                for (int l = 0; l < 32; l++) {
                    const int i = P.row[p0 + l];
                    if (i < 0) continue;
                    const int r0 = ptr[i], d = diag[i], r1 = ptr[i + 1], nlow = d - r0;
                    F.rec[2 * (p0 + l)] = r0;
                    F.rec[2 * (p0 + l) + 1] = nlow | (r1 - 1 - d) << 8;
                    for (int a = r0; a < d; a++) {
                        const int k = col[a], q = W - nlow + (a - r0);
                        int e = a + 1;
                        for (int u = diag[k] + 1; u < ptr[k + 1]; u++) {
                            while (e < r1 && col[e] < col[u]) e++;
                            if (e == r1) break;
                            if (col[e] != col[u]) continue;
                            const int entry = e < d ? W - nlow + (e - r0) : W + (e - d);
                            src[pair_index(W, entry, q)][l] = u;
                        }
                    }
                }
                for (int k = 0; k < NP; k++)
                    for (int l = 0; l < 32; l++) {
                        const int u = src[k][l];
                        if (u < 0) continue;
                        used |= 1u << k;
                        // the row that u belongs to is the lower entry's column
                        int r = 0;
                        {
                            const int i = P.row[p0 + l], d = diag[i];
                            for (int a = ptr[i]; a < d; a++)
                                if (u > diag[col[a]] && u < ptr[col[a] + 1]) r = col[a];
                        }
                        const size_t at = (size_t)c * kPos * NP + (size_t)k * kPos + 32 * (size_t)st + l;
                        const int back = (int)((p0 - lo) / 32) - (pos[r] - lo) / 32;
                        if (pos[r] >= lo && pos[r] < hi && back < P.ring) {
                            F.place[at] = (short)((u - diag[r] - 1) * rw + (pos[r] - lo) % rw);
                        } else {
                            F.place[at] = (short)(W * rw + (int)(x.size() % kSlots));
                            x.push_back(u);
                        }
                    }
            }
            if (x.size() - before > kSlots / 2) bad = 1;
            F.ext_end[c] = (int)x.size();
        }
    }
    if (bad || W * rw + kSlots > 32767) return false;
    for (int s = 0; s < P.strips; s++) F.ext_first[s + 1] = F.ext_first[s] + (int)ext[s].size();
    F.ext.resize(F.ext_first[P.strips]);
    for (int s = 0; s < P.strips; s++) std::copy(ext[s].begin(), ext[s].end(), F.ext.begin() + F.ext_first[s]);
    F.used = used;
    F.width = W;
    return true;
}

}  // namespace strip

// Walks a strip plan on the CPU with the kernel's own rules (one block per strip, a ring of steps, hand-over
// slots filled by helper lanes, every actor advanced in random order), and solves T x = b by it.  Returns 0,
// 1 where no plan is made, or a negative code for a read of something not there, an overwritten slot or a stall.
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "strip_plan.h"

extern "C" int strip_plan_walk(int n, const int* ptr, const int* col, const double* val, const double* dinv, int lower,
                               const double* b, double* x, unsigned seed, int* info) {
    std::vector<int> beg(ptr, ptr + n), end(ptr + 1, ptr + n + 1), lev(n, 0), order(n);
    int nlev = 0;
    for (int t = 0; t < n; t++) {
        const int i = lower ? t : n - 1 - t;
        for (int k = beg[i]; k < end[i]; k++) lev[i] = std::max(lev[i], lev[col[k]] + 1);
        nlev = std::max(nlev, lev[i] + 1);
    }
    std::vector<int> at(nlev + 1, 0);
    for (int i = 0; i < n; i++) at[lev[i] + 1]++;
    for (int l = 0; l < nlev; l++) at[l + 1] += at[l];
    for (int i = 0; i < n; i++) order[at[lev[i]]++] = i;
    strip::Plan P;
    if (!strip::make_plan(P, n, order, lev, nlev, beg, end, col, lower != 0)) return 1;
    info[0] = P.strips;
    info[1] = P.ring;
    info[2] = P.width;
    info[3] = (int)P.ext.size();
    const int slot0 = P.ring * 32, lanes = 32 * strip::kHelpers;
    std::vector<char> have(n, 0), seen(n, 0);
    struct Strip {
        std::vector<double> ops;
        std::vector<char> full;
        std::vector<int> entry;  // each helper lane's entry
        int step = 0, steps = 0;
    };
    std::vector<Strip> S(P.strips);
    for (int s = 0; s < P.strips; s++) {
        S[s].ops.assign(slot0 + strip::kSlots + 1, NAN);
        S[s].ops[slot0 + strip::kSlots] = 0.0;
        S[s].full.assign(slot0 + strip::kSlots + 1, 0);
        S[s].full[slot0 + strip::kSlots] = 1;
        S[s].steps = (P.first[s + 1] - P.first[s]) * strip::kSteps;
        for (int l = 0; l < lanes; l++) S[s].entry.push_back(l);
    }
    std::mt19937 rng(seed);
    long idle = 0;
    int open = P.strips;
    while (open > 0) {
        const int s = (int)(rng() % P.strips);
        Strip& T = S[s];
        bool moved = false;
        const int ne = P.ext_first[s + 1] - P.ext_first[s];
        const int l = (int)(rng() % lanes);
        for (int r = 0; r < lanes; r++) {  // the helper lanes, from a random one on
            int& e = T.entry[(l + r) % lanes];
            if (e >= ne) continue;
            const int src = P.ext[P.ext_first[s] + e], q = slot0 + e % strip::kSlots;
            if (have[src] && !T.full[q]) {
                T.ops[q] = x[src];
                T.full[q] = 1;
                e += lanes;
                moved = true;
            }
        }
        if (T.step < T.steps) {
            const int c = P.first[s] + T.step / strip::kSteps, w = P.table[4 * (size_t)c + 1];
            const size_t p0 = (size_t)c * strip::kPos + 32 * (size_t)(T.step % strip::kSteps);
            const size_t q0 = P.table[4 * (size_t)c] + 32 * (size_t)(T.step % strip::kSteps);
            bool ready = true;
            // a chunk's fetched entries are awaited before its first step
            const int got = T.step < strip::kSteps ? 0 : P.table[4 * (size_t)c - 2], upto = P.table[4 * (size_t)c + 2];
            if (upto < got || upto - got > strip::kSlots / 2) return -7;
            for (int e = got; e < upto && T.step % strip::kSteps == 0; e++) ready = ready && T.full[slot0 + e % strip::kSlots];
            for (int k = 0; k < w && ready; k++)
                for (int lane = 0; lane < 32; lane++) {
                    const int e = P.enc[q0 + (size_t)k * strip::kPos + lane];
                    if (e < 0 || e > slot0 + strip::kSlots) return -1;
                    if (!T.full[e]) return -2;  // a ring entry that was never written, or a slot not awaited
                }
            if (ready) {
                double res[32];
                for (int lane = 0; lane < 32; lane++) {
                    const int i = P.row[p0 + lane];
                    double v = i >= 0 ? b[i] : 0.0;
                    for (int k = 0; k < w; k++) {
                        const size_t q = q0 + (size_t)k * strip::kPos + lane;
                        const int e = P.enc[q], p = P.perm[q];
                        if (i < 0 && p >= 0) return -3;
                        v = std::fma(-(p >= 0 ? val[p] : 0.0), T.ops[e], v);
                    }
                    res[lane] = dinv && i >= 0 ? v * dinv[i] : v;
                }
                for (int lane = 0; lane < 32; lane++) {
                    const int i = P.row[p0 + lane], q = (T.step & (P.ring - 1)) * 32 + lane;
                    T.ops[q] = res[lane];
                    T.full[q] = 1;
                    if (i < 0) continue;
                    if (seen[i]) return -4;
                    seen[i] = have[i] = 1;
                    x[i] = res[lane];
                }
                if (T.step % strip::kSteps == strip::kSteps - 1)
                    for (int e = got; e < upto; e++) T.full[slot0 + e % strip::kSlots] = 0;
                moved = true;
                if (++T.step == T.steps) open--;
            }
        }
        idle = moved ? 0 : idle + 1;
        if (idle > 200000L) return -5;
    }
    for (int i = 0; i < n; i++)
        if (!seen[i]) return -6;
    return 0;
}

// The factorisation by the factor plan, strip after strip: 0, 1 where no plan is made, negative for an operand that
// is not there or is another entry's.
extern "C" int strip_factor_walk(int n, const int* ptr, const int* col, const double* val, double* f, int* info) {
    std::vector<int> beg(n), end(n), diag(n, -1), lev(n, 0), order(n);
    int nlev = 0;
    for (int i = 0; i < n; i++) {
        beg[i] = end[i] = ptr[i];
        for (int k = ptr[i]; k < ptr[i + 1]; k++) {
            if (col[k] == i) diag[i] = k;
            if (col[k] < i) {
                end[i] = k + 1;
                lev[i] = std::max(lev[i], lev[col[k]] + 1);
            }
        }
        nlev = std::max(nlev, lev[i] + 1);
    }
    std::vector<int> at(nlev + 1, 0);
    for (int i = 0; i < n; i++) at[lev[i] + 1]++;
    for (int l = 0; l < nlev; l++) at[l + 1] += at[l];
    for (int i = 0; i < n; i++) order[at[lev[i]]++] = i;
    strip::Plan P;
    strip::FactorPlan F;
    if (!strip::make_plan(P, n, order, lev, nlev, beg, end, col, true)) return 1;
    if (!strip::make_factor_plan(F, P, n, ptr, col, diag)) return 1;
    const int W = F.width, NP = strip::pairs_of(W), rw = P.ring * 32;
    info[0] = P.strips;
    info[1] = W;
    info[2] = (int)F.ext.size();
    std::vector<char> have(ptr[n], 0);
    for (int s = 0; s < P.strips; s++) {
        std::vector<double> ops(W * rw + strip::kSlots, NAN);
        std::vector<char> full(W * rw + strip::kSlots, 0);
        int filled = 0;
        for (int step = 0; step < (P.first[s + 1] - P.first[s]) * strip::kSteps; step++) {
            const int c = P.first[s] + step / strip::kSteps;
            if (step % strip::kSteps == 0) {
                if (F.ext_end[c] - filled > strip::kSlots / 2) return -3;
                for (; filled < F.ext_end[c]; filled++) {
                    const int u = F.ext[F.ext_first[s] + filled], q = W * rw + filled % strip::kSlots;
                    if (!have[u]) return -4;
                    ops[q] = f[u];
                    full[q] = 1;
                }
            }
            std::vector<double> v(32 * (2 * W + 1), 0.0);
            for (int l = 0; l < 32; l++) {
                const size_t p = (size_t)c * strip::kPos + 32 * (size_t)(step % strip::kSteps) + l;
                double* x = &v[l * (2 * W + 1)];
                const int r0 = F.rec[2 * p], nlow = F.rec[2 * p + 1] & 0xff, nup = F.rec[2 * p + 1] >> 8;
                if ((r0 >= 0) != (P.row[p] >= 0)) return -5;
                for (int e = 0; e < 2 * W + 1; e++) {
                    const int k = e - (W - nlow);
                    x[e] = r0 >= 0 && k >= 0 && k <= nlow + nup ? val[r0 + k] : e == W ? 1.0 : 0.0;
                }
                for (int e = 0; e < 2 * W + 1; e++) {
                    double sum = 0.0;
                    for (int q = 0; q < W && q < e; q++) {
                        const int k = strip::pair_index(W, e, q);
                        const int a = F.place[(size_t)c * strip::kPos * NP + (size_t)k * strip::kPos + 32 * (size_t)(step % strip::kSteps) + l];
                        if (a < 0) continue;
                        if (!(F.used >> k & 1u) || r0 < 0) return -6;
                        if (!full[a]) return -7;
                        const double t = x[q] * ops[a];
                        sum = sum + t;
                    }
                    x[e] = x[e] - sum;
                }
                for (int t = 0; t < W; t++) x[W + 1 + t] /= x[W];
                if (r0 < 0) continue;
                for (int k = 0; k <= nlow + nup; k++) {
                    f[r0 + k] = x[k + W - nlow];
                    have[r0 + k] = 1;
                }
            }
            for (int l = 0; l < 32; l++)
                for (int t = 0; t < W; t++) {
                    const int q = t * rw + (step * 32 + l) % rw;
                    ops[q] = v[l * (2 * W + 1) + W + 1 + t];
                    full[q] = 1;
                }
        }
    }
    return 0;
}

// a / d by two corrections with the rounded reciprocal: how many of the count random pairs round otherwise than
// the division
extern "C" long quotient_misses(long count, unsigned seed) {
    std::mt19937_64 rng(seed);
    long bad = 0;
    for (long k = 0; k < count; k++) {
        auto draw = [&] {
            uint64_t m = rng() & 0xfffffffffffffull;
            switch (rng() % 8) {  // mantissas at the ends of their range among them
                case 0: m &= 7; break;
                case 1: m |= 0xffffffffffff8ull; break;
                default: break;
            }
            const uint64_t u = (rng() & 1) << 63 | (uint64_t)(1023 - 400 + rng() % 801) << 52 | m;
            double x;
            memcpy(&x, &u, 8);
            return x;
        };
        const double a = draw(), d = draw(), r = 1.0 / d;
        const double q0 = a * r, q1 = std::fma(std::fma(-d, q0, a), r, q0), q = std::fma(std::fma(-d, q1, a), r, q1);
        if (q != a / d) bad++;
    }
    return bad;
}

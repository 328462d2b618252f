// Walks a strip plan on the CPU with the kernel's own rules (one block per strip, a ring of steps, hand-over
// slots filled by helper lanes, every actor advanced in random order), and solves T x = b by it.  Returns 0,
// 1 where no plan is made, or a negative code for a read of something not there, an overwritten slot or a stall.
#include <cmath>
#include <cstdlib>
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

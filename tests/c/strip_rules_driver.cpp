// Which solve a triangular factor takes (strip_plan.h): the strips' plan, its estimates and the choice by them; and
// the row recurrence, each product and sum rounded as one fused operation.
#include <cmath>
#include <vector>

#include "strip_plan.h"

// out: strips, entries per row where fixed, most entries, estimated ns of the strips and of the one block in FP32, FP64
extern "C" int strip_rules(int n, const int* ptr, const int* col, int lower, double* out) {
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
    if (!strip::make_plan(P, n, order, lev, nlev, beg, end, col, lower != 0)) return -1;
    const double v[] = {double(P.strips), double(P.width), double(P.max_width), P.ns32, P.win32, P.ns64, P.win64};
    for (int k = 0; k < 7; k++) out[k] = v[k];
    return (strip::pays(P, false) ? 1 : 0) | (strip::pays(P, true) ? 2 : 0);
}

template <typename T>
static void recurrence(int n, const int* ptr, const int* col, const T* val, const T* dinv, int lower, const T* b, T* x) {
    for (int t = 0; t < n; t++) {
        const int i = lower ? t : n - 1 - t;
        T s = b[i];
        for (int p = ptr[i]; p < ptr[i + 1]; p++) s = std::fma(-val[p], x[col[p]], s);
        x[i] = dinv ? s * dinv[i] : s;
    }
}

extern "C" void recurrence64(int n, const int* ptr, const int* col, const double* val, const double* dinv, int lower,
                             const double* b, double* x) {
    recurrence(n, ptr, col, val, dinv, lower, b, x);
}
extern "C" void recurrence32(int n, const int* ptr, const int* col, const float* val, const float* dinv, int lower,
                             const float* b, float* x) {
    recurrence(n, ptr, col, val, dinv, lower, b, x);
}

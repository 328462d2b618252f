// strip_factor.cuh - ILU(0) pipelined over the strips of the lower factor's plan (strip_solve.cuh).
//
// The walking warps take 32 rows of one level at a time, a lane per row.  A row's operands U_kj come from the
// ring of the last steps' upper entries in shared memory or from a slot a helper warp fills; its sums
// take the products L_ik U_kj in ascending k, each product and sum rounded by itself, as the other
// factorisation of this library does, so the factors are equal to its bit for bit.  What bounds a step is a
// chain of FP64 operations of 64 cycles each, dependent or not: the lower entries in turn, the diagonal's
// sum, a reciprocal and a division.  So the entries right of the diagonal are formed by warps of their own:
// AT2 damage, 513 x 513 nodes (1,025 levels), GB300: the row pool 13.8 ms, one walking warp 2.1 ms, a
// warp for the diagonal and one per upper entry 1.25 ms; 1,025 x 1,025 nodes 29 -> 2.6 ms.
#pragma once

#include "strip_solve.cuh"

namespace strip {

// a / d with r = 1 / d rounded to nearest
__device__ __forceinline__ double quotient(double a, double d, double r) {
    const unsigned ha = (unsigned)__double2hiint(a);
    const bool zero = ((ha << 1) | (unsigned)__double2loint(a)) == 0;
    if (mid_range((unsigned)__double2hiint(d)) && (zero || mid_range(ha))) {
        const double q0 = a * r;
        const double q1 = __fma_rn(__fma_rn(-d, q0, a), r, q0);
        const double q2 = __fma_rn(__fma_rn(-d, q1, a), r, q1);
        return zero ? q0 : q2;
    }
    return __ddiv_rn(a, d);
}

// -0 becomes +0 (by its bits)
__device__ __forceinline__ double plus_zero(double t) {
    return ((unsigned)__double2loint(t) | ((unsigned)__double2hiint(t) ^ 0x80000000u)) == 0 ? 0.0 : t;
}

struct FactorArgs {
    int ring, stages;
    unsigned used;             // pairs some row has
    const int* first;          // first chunk of each strip
    const int* ext_first;      // first fetched entry of each strip
    const int* ext;            // CSR entry of each fetched entry
    const int* ext_end;        // per chunk
    const int2* rec;           // per position: first CSR entry, lower | upper << 8 ((-1, 0) without a row)
    const short* place;        // per chunk and pair
    const double* a;           // per chunk and entry (W lower, diagonal, W upper): A's values, no NaN but the canonical
    double* f;                 // CSR entry -> factor value, the pending pattern on entry
    unsigned* ticket;
    int* err;                  // 1 a wait ran out, 2 zero pivot
    unsigned long long limit_ns;  // of every wait
};

struct FactorStage {
    int rec, place, a, bytes;
};
__host__ __device__ constexpr FactorStage factor_stage(int W) {
    return FactorStage{0, 8 * kPos, 8 * kPos + 2 * kPos * pairs_of(W),
                       8 * kPos + 2 * kPos * pairs_of(W) + 8 * kPos * (2 * W + 1)};
}
__host__ __device__ inline int factor_operand_bytes(int W, int ring) { return ((W * ring * 32 + kSlots) * 8 + 127) / 128 * 128; }
inline size_t factor_smem(int W, int ring, int stages) {
    return (size_t)kHead + 512 + factor_operand_bytes(W, ring) + (size_t)stages * factor_stage(W).bytes;
}
inline int factor_stages(int W, int ring) {
    int s = 6;
    while (s > 1 && factor_smem(W, ring, s) > (size_t)kSmemMax) s--;
    return s;
}

// 1 + W warps walk the strip together, on different FP64 units where they can: each forms the rows' lower entries
// for itself, warp 0 the diagonal and its reciprocal, warp 1 + t the t-th upper entry; the copying warp and the
// helpers follow.
__host__ __device__ constexpr int factor_threads(int W) { return 32 * (1 + W + 1 + kHelpers); }

// a barrier of the walking warps
template <int W>
__device__ __forceinline__ void walkers_sync() {
    asm volatile("barrier.cta.sync 1, %0;" ::"n"(32 * (1 + W)) : "memory");
}
template <int W>
__device__ __forceinline__ bool walkers_all(bool ok) {
    int all;
    asm volatile(
        "{\n .reg .pred P, Q;\n setp.ne.s32 P, %1, 0;\n barrier.cta.red.and.pred Q, 1, %2, P;\n selp.s32 %0, 1, 0, "
        "Q;\n}"
        : "=r"(all)
        : "r"((int)ok), "n"(32 * (1 + W))
        : "memory");
    return all != 0;
}

template <int W>
__global__ void __launch_bounds__(factor_threads(W), 1) factor_kernel(const FactorArgs a) {
    using B = Bits<double>;
    using U = B::U;
    constexpr int NP = pairs_of(W), NE = 2 * W + 1, NL = W * (W - 1) / 2;
    constexpr FactorStage L = factor_stage(W);
    extern __shared__ __align__(128) unsigned char strip_smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(strip_smem);
    volatile int* ctl = reinterpret_cast<volatile int*>(strip_smem + 64);
    double2* pivot = reinterpret_cast<double2*>(strip_smem + kHead);  // the rows' diagonals and reciprocals
    unsigned char* ops = strip_smem + kHead + 512;                    // W rings of upper entries, then the slots
    unsigned char* stages = strip_smem + kHead + 512 + factor_operand_bytes(W, a.ring);
    const int rw = a.ring * 32;
    unsigned char* slots = ops + W * rw * 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        ctl[0] = (int)atomicAdd(a.ticket, 1u);
        ctl[1] = 0;
        for (int k = 0; k < a.stages; k++) bulk::mbar_init(bars + k);
        bulk::fence_mbar_init();
    }
    for (int k = threadIdx.x; k < kSlots; k += factor_threads(W)) put<double>(slots + 8 * k, B::kPending);
    __syncthreads();
    const int strip = ctl[0];
    const int c0 = __ldg(a.first + strip), c1 = __ldg(a.first + strip + 1);
    if (warp > W + 1) {
        fetch_entries<double>(a.f, a.ext, __ldg(a.ext_first + strip), __ldg(a.ext_first + strip + 1),
                              threadIdx.x - 32 * (W + 2), slots, a.err, a.limit_ns);
        return;
    }
    if (warp == W + 1) {
        if (lane != 0) return;
        copy_chunks(c0, c1, a.stages, L.bytes, stages, bars, ctl + 1, a.err, a.limit_ns, [&](int c, unsigned char* st, uint64_t* bar) {
            bulk::mbar_expect_tx(bar, (unsigned)L.bytes);
            bulk::copy(st + L.rec, a.rec + (size_t)c * kPos, 8u * kPos, bar);
            bulk::copy(st + L.place, a.place + (size_t)c * kPos * NP, 2u * kPos * NP, bar);
            bulk::copy(st + L.a, a.a + (size_t)c * kPos * NE, 8u * kPos * NE, bar);
        });
        return;
    }
    // this warp's entry: the diagonal, or an upper entry
    const int own = W + warp;
    const unsigned own_used = a.used >> (NL + warp * W);
    const int chunks = c1 - c0;
    int place = lane;  // this step's entries in the rings
    int got = 0, end = __ldg(a.ext_end + c0), end1 = chunks > 1 ? __ldg(a.ext_end + c0 + 1) : 0;
    U first = B::kPending;
    int stage = 0;
    unsigned phase = 0;
    // v - sum of the pairs: products in ascending q, a pair the row does not have takes no part (L may be infinite).
    // A warp issues an FP64 operation in 64 cycles whether or not it depends on the one before, so what no row
    // needs is branched around.
    auto reduced = [&](double v, const double (&low)[W], const int* at, const U* u, unsigned used, int n) {
        double s = 0.0;
        bool open = true;  // no product before: 0 + t is t, and +0 for t = -0
#pragma unroll
        for (int q = 0; q < W; q++) {
            if (q < n && (used >> q & 1u)) {
                const double t = __dmul_rn(low[q], B::value(u[q]));
                const double sum = open ? plus_zero(t) : __dadd_rn(s, t);
                s = at[q] >= 0 ? sum : s;
                open = false;
            }
        }
        return open ? v : __dsub_rn(v, s);
    };
    for (int c = 0; c < chunks; c++) {
        const unsigned char* st = stages + stage * L.bytes;
        bool ok = bulk::mbar_wait(bars + stage, phase, a.err, 1);
        ok = await_entries<double>(got, end, first, slots, lane, a.err, a.limit_ns) && ok;
        if (!walkers_all<W>(ok)) break;
        for (int i = 0; i < kSteps; i++) {
            const int p = 32 * i + lane;
            const int2 rec = reinterpret_cast<const int2*>(st + L.rec)[p];
            const int nlow = rec.y & 0xff, nup = rec.y >> 8;
            const short* pl = reinterpret_cast<const short*>(st + L.place) + p;
            const double* av = reinterpret_cast<const double*>(st + L.a) + p;
            int at[NL + W];
            U u[NL + W];
#pragma unroll
            for (int k = 0; k < NL + W; k++) at[k] = pl[(k < NL ? k : k + warp * W) * kPos];
#pragma unroll
            for (int k = 0; k < NL + W; k++) u[k] = get<double>(ops + 8 * (at[k] >= 0 ? at[k] : 0));
            double low[W];
#pragma unroll
            for (int q = 0; q < W; q++) {
                low[q] = reduced(av[q * kPos], low, at + q * (q - 1) / 2, u + q * (q - 1) / 2, a.used >> (q * (q - 1) / 2), q);
            }
            const double x = reduced(av[own * kPos], low, at + NL, u + NL, own_used, W);
            double* f = a.f + rec.x;
            if (warp == 0) {
                const double r = __drcp_rn(x);
                pivot[lane] = make_double2(x, r);
                // a zero pivot fails the factorisation where a quotient needs it
                if (nup > 0 && (U(__double_as_longlong(x)) << 1) == 0) atomicExch(a.err, 2);
                walkers_sync<W>();
                if (rec.x >= 0) f[nlow] = x;
#pragma unroll
                for (int q = 0; q < W; q++) {
                    const int e = q - (W - nlow);  // the row's e-th lower entry
                    if (e >= 0) f[e] = low[q];
                }
            } else {
                const int t = warp - 1;
                walkers_sync<W>();
                const double2 d = pivot[lane];
                const U w = U(__double_as_longlong(quotient(x, d.x, d.y)));
                put<double>(ops + 8 * (t * rw + place), w);
                B::publish(a.f + (t < nup ? rec.x + nlow + 1 + t : 0), t < nup, w);
            }
            place = (place + 32) & (rw - 1);
            if (i == kSteps - 2)
                first = end + lane < end1 ? get<double>(slots + (end + lane) % kSlots * 8) : U(0);
            walkers_sync<W>();  // the step's entries are in the rings before the next one's reads
        }
        if (warp == 0) {
            for (int e = got + lane; e < end; e += 32) put<double>(slots + e % kSlots * 8, B::kPending);
            if (lane == 0) ctl[1] = c + 1;
        }
        got = end;
        end = end1;
        end1 = c + 2 < chunks ? __ldg(a.ext_end + c0 + c + 2) : 0;
        if (++stage == a.stages) {
            stage = 0;
            phase ^= 1u;
        }
    }
}

}  // namespace strip

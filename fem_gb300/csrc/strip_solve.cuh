// strip_solve.cuh - triangular solves pipelined over strips of rows.
//
// A sparse triangular solve is a chain of levels; on mesh matrices there are thousands, each a few
// hundred to a few thousand rows wide.  Here the rows are cut into contiguous strips (in the order of
// the recurrence: ascending indices for a lower factor, descending for an upper one), a block per
// strip on an SM of its own.  A strip walks its own levels in steps of at most 32 rows of one level,
// a lane per row, with nothing but a __syncwarp between steps: the solution entries of its last
// `ring` steps are read back from shared memory.  Entries that come from another strip (or from
// further back) are fetched by two helper warps, which poll the solution in global memory (filled
// with a NaN pattern that arithmetic does not produce) far ahead of the walking warp and hand the
// values over in slots of shared memory that hold the same pattern while empty; the walking warp awaits them
// a chunk of eight steps at a time (step by step, the test and its branch cost more than the products: 1,025 x
// 1,025 nodes, FP32, a wait per 8 steps 0.25 ms, per 4 steps 0.28 ms, per step 0.30 ms a solve).  A fourth warp copies
// the steps' rows, right-hand sides, sources and factor values into shared memory with bulk copies, a
// chunk of eight steps per stage, several stages ahead.
//
// So a level costs the walking warp the latency of one shared-memory read, its products and one store,
// and the strips follow one another at the distance of one exchange through L2.  What bounds it is that
// chain: levels x step + strips x exchange.  Measured on GB300 (three entries a row): a step 63 ns in FP32
// and 198 ns in FP64 (an FP64 operation takes 64 cycles), 77 and 209 ns with entries from a neighbouring
// strip; an exchange 2.0 to 2.8 us.  30 rows of the widest level a strip: with 15, the second term made the
// 1,025 x 1,025 solve 23 % slower, with 60 the first one 55 %.
//
// Progress: a strip needs strips before it only, and blocks take strips in the order in which they
// start (a ticket), so every awaited strip is running.  Within a strip a helper lane takes its entries in
// step order; an entry waits for a row of an earlier step or strip and for its slot, which an earlier
// step empties.  Every wait is bounded.  Products are subtracted in the factor's entry order, as the
// other solves of this library do, so the results are equal to theirs bit for bit.
#pragma once

#include <cstdint>

#include "bulk_copy.cuh"
#include "strip_plan.h"

namespace strip {

// ---------------------------------------------------------------- device side
template <typename T>
struct Bits;
template <>
struct Bits<float> {
    using U = unsigned;
    static constexpr U kPending = 0xffffffffu;  // a NaN arithmetic does not produce
    static __device__ __forceinline__ U of(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float value(U u) { return __uint_as_float(u); }
    // the solution's entries are read by other blocks while the kernel runs
    static __device__ __forceinline__ void publish(float* p, bool on, U u) {
        asm volatile("{\n .reg .pred P;\n setp.ne.s32 P, %2, 0;\n @P st.relaxed.gpu.global.u32 [%0], %1;\n}" ::"l"(p),
                     "r"(u), "r"((int)on)
                     : "memory");
    }
    static __device__ __forceinline__ U poll(const float* p) {
        U u;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(u) : "l"(p) : "memory");
        return u;
    }
};
template <>
struct Bits<double> {
    using U = unsigned long long;
    static constexpr U kPending = 0xffffffffffffffffull;
    static __device__ __forceinline__ U of(double v) { return (U)__double_as_longlong(v); }
    static __device__ __forceinline__ double value(U u) { return __longlong_as_double((long long)u); }
    static __device__ __forceinline__ void publish(double* p, bool on, U u) {
        asm volatile("{\n .reg .pred P;\n setp.ne.s32 P, %2, 0;\n @P st.relaxed.gpu.global.u64 [%0], %1;\n}" ::"l"(p),
                     "l"(u), "r"((int)on)
                     : "memory");
    }
    static __device__ __forceinline__ U poll(const double* p) {
        U u;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
        return u;
    }
};

// a word of the ring or a slot, in shared memory
template <typename TX>
__device__ __forceinline__ typename Bits<TX>::U get(const unsigned char* p) {
    return *reinterpret_cast<const volatile typename Bits<TX>::U*>(p);
}
template <typename TX>
__device__ __forceinline__ void put(unsigned char* p, typename Bits<TX>::U u) {
    *reinterpret_cast<volatile typename Bits<TX>::U*>(p) = u;
}

// one load each: what a row's entry and a position hold
template <typename TX>
struct Entry;
template <>
struct __align__(8) Entry<float> {
    unsigned place;
    float val;  // 0 on padding
};
template <>
struct __align__(16) Entry<double> {
    unsigned place, pad;
    double val;
};
template <typename TX>
struct Point;
template <>
struct __align__(8) Point<float> {
    int row;  // -1: none
    float dinv;
};
template <>
struct __align__(16) Point<double> {
    int row, pad;
    double dinv;
};

template <typename TX>
struct Args {
    int ring, max_width, stages;
    const int* first;       // first chunk of each strip
    const int* ext_first;   // first fetched entry of each strip
    const int* ext;         // row of each fetched entry
    const int4* table;      // chunk -> (offset of its entries, entries per row, end of its fetched entries, 0)
    // the operands: no NaN among them but the canonical one
    const Entry<TX>* entry;  // entry -> place of its operand in shared memory (bytes) and factor value
    const Point<TX>* point;  // position -> row and 1 / diagonal
    const TX* b;             // position -> right-hand side
    TX* x;                  // row -> solution, the pending pattern on entry
    unsigned* ticket;       // strips taken, 0 on entry
    int* err;
    unsigned long long limit_ns;  // of every wait
};

// byte offsets inside a stage, for chunks of up to `width` entries per row
struct Stage {
    int point, b, entry, bytes;
};
__host__ __device__ inline Stage stage_layout(int width, int tx) {
    Stage s;
    s.point = 0;
    s.b = 2 * tx * kPos;
    s.entry = s.b + tx * kPos;
    s.bytes = s.entry + 2 * tx * kPos * width;
    return s;
}
constexpr int kHead = 128;  // barriers, the strip and the chunk counter
__host__ __device__ inline int operand_bytes(int ring, int tx) { return ((ring * 32 + kSlots + 1) * tx + 127) / 128 * 128; }
inline size_t smem_bytes(int ring, int width, int tx, int stages) {
    return (size_t)kHead + operand_bytes(ring, tx) + (size_t)stages * stage_layout(width, tx).bytes;
}
inline int stages_for(int ring, int width, int tx) {
    int s = 6;
    while (s > 2 && smem_bytes(ring, width, tx, s) > (size_t)kSmemMax) s--;
    return s;
}

// after a failed poll: every 64th looks at the error word and the clock (a read of either costs as much as
// the wait); false: give up (after limit_ns)
__device__ __forceinline__ bool keep_waiting(long& polls, unsigned long long& t0, int* err, int code,
                                             unsigned long long limit_ns) {
    if ((++polls & 63) != 0) return true;
    if (polls == 64) t0 = bulk::device_ns();
    if (polls > bulk::kWaitPolls || *(volatile int*)err || bulk::device_ns() - t0 > limit_ns) {
        atomicCAS(err, 0, code);
        return false;
    }
    return true;
}

// the helper warps: fetched entry e of the strip goes to slot e mod kSlots once its row is solved and the
// slot is empty.  One loop for all lanes, each at an entry of its own: a lane that waits holds up no other.
template <typename TX>
__device__ void fetch_entries(const TX* x, const int* __restrict__ ext, int e0, int e1, int lane, unsigned char* slots,
                              int* err, unsigned long long limit_ns) {
    using B = Bits<TX>;
    using U = typename B::U;
    int e = e0 + lane;
    int src = e < e1 ? __ldg(ext + e) : 0;
    int nsrc = e + 32 * kHelpers < e1 ? __ldg(ext + e + 32 * kHelpers) : 0;
    U u = B::kPending;
    long polls = 0;
    unsigned long long t0 = 0;
    while (e < e1) {
        unsigned char* slot = slots + (e - e0) % kSlots * (int)sizeof(TX);
        if (u == B::kPending) u = B::poll(x + src);
        if (u != B::kPending && get<TX>(slot) == B::kPending) {
            put<TX>(slot, u);
            u = B::kPending;
            e += 32 * kHelpers;
            src = nsrc;
            nsrc = e + 32 * kHelpers < e1 ? __ldg(ext + e + 32 * kHelpers) : 0;
            polls = 0;
        } else if (!keep_waiting(polls, t0, err, 1, limit_ns)) {
            return;
        }
    }
}

// the walking warp: the fetched entries [got, end) of a chunk are there (false: given up).  first: one of them
// per lane, looked at before; where all were there and they are at most 32, nothing is waited for.
template <typename TX>
__device__ __forceinline__ bool await_entries(int got, int end, typename Bits<TX>::U first, const unsigned char* slots,
                                              int lane, int* err, unsigned long long limit_ns) {
    bool ok = true;
    if (end - got > 32 || __any_sync(0xffffffffu, first == Bits<TX>::kPending)) {
        for (int e = got + lane; e < end; e += 32) {
            const unsigned char* slot = slots + e % kSlots * (int)sizeof(TX);
            long polls = 0;
            unsigned long long t0 = 0;
            while (ok && get<TX>(slot) == Bits<TX>::kPending) ok = keep_waiting(polls, t0, err, 1, limit_ns);
        }
        __syncwarp();
    }
    return ok;
}

// the copying warp's lane: chunk c of the strip's c0 .. c1 into stage (c - c0) mod S once the walking warp is done
// with chunk c - S; issue(c, stage, barrier) announces the chunk's bytes and starts its copies
template <typename F>
__device__ __forceinline__ void copy_chunks(int c0, int c1, int S, int stage_bytes, unsigned char* stages, uint64_t* bars,
                                            const volatile int* done, int* err, unsigned long long limit_ns, F issue) {
    int c = c0;
    for (; c < c1; c++) {
        long polls = 0;
        unsigned long long t0 = 0;
        bool ok = true;
        while (ok && *done < c - c0 - S + 1) ok = keep_waiting(polls, t0, err, 1, limit_ns);
        if (!ok) break;
        bulk::fence_proxy_async();  // the stage was last read through ordinary loads
        issue(c, stages + ((c - c0) % S) * stage_bytes, bars + (c - c0) % S);
    }
    // no copy may still be landing when the block exits, also where the walking warp gave up
    for (int k = c - S > c0 ? c - S : c0; k < c; k++)
        bulk::mbar_drain(bars + (k - c0) % S, (unsigned)(((k - c0) / S) & 1));
}

// EM > 0: every row has EM entries (padded), held in registers and loaded a step ahead; 0: the entries of
// each chunk's rows counted in the table and read where they are used.  DINV: rows are scaled by 1 / diagonal.
template <typename TX, int EM, bool DINV>
__global__ void __launch_bounds__(kThreads, 1) solve_kernel(const Args<TX> a) {
    using B = Bits<TX>;
    using U = typename B::U;
    extern __shared__ __align__(128) unsigned char strip_smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(strip_smem);
    volatile int* ctl = reinterpret_cast<volatile int*>(strip_smem + 64);  // [0] strip, [1] chunks walked
    unsigned char* stages = strip_smem + kHead + operand_bytes(a.ring, sizeof(TX));
    unsigned char* ops = strip_smem + kHead;  // the ring, the slots, a zero
    unsigned char* slots = ops + a.ring * 32 * (int)sizeof(TX);
    const Stage L = stage_layout(a.max_width, sizeof(TX));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        ctl[0] = (int)atomicAdd(a.ticket, 1u);
        ctl[1] = 0;
        for (int k = 0; k < a.stages; k++) bulk::mbar_init(bars + k);
        bulk::fence_mbar_init();
        put<TX>(slots + kSlots * sizeof(TX), U(0));
    }
    for (int k = threadIdx.x; k < kSlots; k += kThreads) put<TX>(slots + k * sizeof(TX), B::kPending);
    __syncthreads();
    const int strip = ctl[0];
    const int c0 = __ldg(a.first + strip), c1 = __ldg(a.first + strip + 1);
    if (warp >= 2) {
        fetch_entries<TX>(a.x, a.ext, __ldg(a.ext_first + strip), __ldg(a.ext_first + strip + 1), threadIdx.x - 64, slots,
                          a.err, a.limit_ns);
        return;
    }
    if (warp == 1) {
        if (lane != 0) return;
        copy_chunks(c0, c1, a.stages, L.bytes, stages, bars, ctl + 1, a.err, a.limit_ns, [&](int c, unsigned char* st, uint64_t* bar) {
            const int4 tb = __ldg(a.table + c);
            const unsigned pb = (unsigned)sizeof(TX) * kPos;
            bulk::mbar_expect_tx(bar, pb * (3u + 2u * tb.y));
            bulk::copy(st + L.point, a.point + (size_t)c * kPos, 2u * pb, bar);
            bulk::copy(st + L.b, a.b + (size_t)c * kPos, pb, bar);
            if (tb.y) bulk::copy(st + L.entry, a.entry + tb.x, 2u * pb * tb.y, bar);
        });
        return;
    }
    constexpr int W = EM > 0 ? EM : 1;
    struct Row {
        Point<TX> p;
        TX b;
        Entry<TX> e[W];
    };
    auto load = [&](Row& r, const unsigned char* st, int p) {
        r.p = reinterpret_cast<const Point<TX>*>(st + L.point)[p];
        r.b = reinterpret_cast<const TX*>(st + L.b)[p];
        if constexpr (EM > 0) {
#pragma unroll
            for (int k = 0; k < EM; k++) r.e[k] = reinterpret_cast<const Entry<TX>*>(st + L.entry)[k * kPos + p];
        }
    };
    auto scaled = [&](const Row& r, TX v) {
        if constexpr (DINV) return v * r.p.dinv;
        return v;
    };
    const int chunks = c1 - c0;
    const unsigned ring_mask = (unsigned)(a.ring * 32 * sizeof(TX)) - 1u;
    unsigned place = lane * (unsigned)sizeof(TX);  // this step's entry in the ring
    int got = 0;                                   // fetched entries of the chunks before
    int end = __ldg(a.table + c0).z, end1 = chunks > 1 ? __ldg(a.table + c0 + 1).z : 0;  // of this chunk and the next
    U first = B::kPending;  // a fetched entry of the chunk, looked at a step early
    unsigned char* st = stages;
    int stage = 0;
    unsigned phase = 0;
    bool ok = bulk::mbar_wait(bars, 0, a.err, 1);
    if (!__all_sync(0xffffffffu, ok)) return;
    Row r[2];
    if constexpr (EM > 0) load(r[0], st, lane);
    for (int c = 0; c < chunks; c++) {
        unsigned char* next = st + L.bytes;
        int nstage = stage + 1;
        unsigned nphase = phase;
        if (nstage == a.stages) {
            next = stages;
            nstage = 0;
            nphase ^= 1u;
        }
        const int w = EM > 0 ? EM : __ldg(a.table + c0 + c).y;
        ok = await_entries<TX>(got, end, first, slots, lane, a.err, a.limit_ns) && ok;
#pragma unroll
        for (int i = 0; i < kSteps; i++) {
            U res;
            int row;
            if constexpr (EM > 0) {
                const Row& cur = r[i & 1];
                U u[W];
#pragma unroll
                for (int k = 0; k < EM; k++) u[k] = get<TX>(ops + cur.e[k].place);
                // the next step's row while these are on their way
                if (i + 1 < kSteps) {
                    load(r[(i + 1) & 1], st, 32 * (i + 1) + lane);
                } else if (c + 1 < chunks) {
                    ok = bulk::mbar_wait(bars + nstage, nphase, a.err, 1) && ok;
                    load(r[0], next, lane);
                }
                TX s = cur.b;
#pragma unroll
                for (int k = 0; k < EM; k++) s -= cur.e[k].val * B::value(u[k]);
                // the operands hold no NaN but the canonical one, so the outcome is not the pending pattern
                res = B::of(scaled(cur, s));
                row = cur.p.row;
            } else {
                const int p = 32 * i + lane;
                load(r[0], st, p);
                TX s = r[0].b;
                for (int k = 0; k < w; k++) {
                    const Entry<TX> e = reinterpret_cast<const Entry<TX>*>(st + L.entry)[k * kPos + p];
                    s -= e.val * B::value(get<TX>(ops + e.place));
                }
                res = B::of(scaled(r[0], s));
                row = r[0].p.row;
            }
            put<TX>(ops + place, res);
            B::publish(a.x + (row >= 0 ? row : 0), row >= 0, res);
            place = (place + 32u * (unsigned)sizeof(TX)) & ring_mask;
            __syncwarp();  // the step's shared-memory accesses come before the next one's
            if (i == kSteps - 2)
                first = end + lane < end1 ? get<TX>(slots + (end + lane) % kSlots * (int)sizeof(TX)) : U(0);
        }
        // the chunk's slots are empty again
        for (int e = got + lane; e < end; e += 32) put<TX>(slots + e % kSlots * (int)sizeof(TX), B::kPending);
        got = end;
        end = end1;
        end1 = c + 2 < chunks ? __ldg(a.table + c0 + c + 2).z : 0;
        if constexpr (EM == 0)
            if (c + 1 < chunks) ok = bulk::mbar_wait(bars + nstage, nphase, a.err, 1) && ok;
        if (!__all_sync(0xffffffffu, ok)) break;
        if (lane == 0) ctl[1] = c + 1;
        st = next;
        stage = nstage;
        phase = nphase;
    }
}

}  // namespace strip

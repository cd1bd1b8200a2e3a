// song_gt.cu -- exact k nearest neighbours on the tensor cores (the ground
// truth that recall is measured against).
//
// The reference computes ground truth by sequential brute force on the CPU
// (bench_cpu.cpp:158-175, a max-heap of the k smallest squared L2 distances
// per query) or in numpy (run_compare.py:199-213).  Here every distance is
// |q|^2 - 2 q.b + |b|^2 with the cross term from 3xBF16 split products on
// the tensor cores: x = hi + lo with hi = bf16(x) and lo = bf16(x - hi), and
// q.b ~= hi_q.hi_b + hi_q.lo_b + lo_q.hi_b accumulated in FP32 (lo.lo is
// below FP32 resolution).  A product whose lo operand is zero everywhere is
// skipped; for integer data in [0, 255] both lo parts are zero and, for
// dim <= 128, every sum stays an integer below 2^24, so distances are exact.
// The squared norms are FP64 sums rounded to FP32 and the distance is formed
// as (|q|^2 - 2 q.b) + |b|^2 in FP32.
//
// Layout in HBM: base and query rows are converted once into BF16 blocks of
// 128 rows x 32 dimensions (8 KB, the tensor cores' shared-memory operand
// layout: K-major, no swizzle, 8 x 16-byte core matrices; core matrices
// adjacent along K are 128 B apart, groups of 8 rows 512 B apart):
// [tile][hi, lo][chunk][128 x 32].
//
// One CTA owns MT x 128 queries (MT = 2 unless that pads too many) and a
// contiguous range of base tiles (a split); warps have fixed roles:
//   a copier brings the queries' blocks into shared memory once, where they
//           fit, then the bases' blocks of each tile through a ring of 32 KB
//           stages (cp.async.bulk, completion counted on mbarriers);
//   an issuer (one thread) issues tcgen05.mma kind::f16 (BF16 x BF16 ->
//           FP32, M = N = 128, K = 16) of every base block against the MT
//           query tiles into one of two sets of MT accumulators in TMEM;
//   4 * MT epilogue warps read the other set (tcgen05.ld, TMEM lane =
//           query, the next 32 columns in flight while these are used).
// What bounds it: with 128 dimensions a tile of 256 x 128 is 1,024 cycles of
// tensor work and 32 KB of base blocks (32 bytes per cycle per SM from L2;
// one query tile per CTA would need 64, more than L2 gives all SMs), and the
// epilogue's 32,768 keys must cost less than that, so a key costs one FMA,
// a quarter of a shared load and one minimum: |b|^2 - 2 q.b against the
// query's threshold (less its |q|^2, widened by more than the rounding
// differences).  Only a 32-column chunk with a key below it forms exact
// distances.  Those below the threshold are appended to the query's list for
// this split in global memory (fire and forget); a list that fills up is cut
// by its warp to its k smallest keys, the k-th becoming the threshold.  A
// query's splits share their smallest threshold through one word per query
// in global memory: any split's k-th distance bounds the final one (and, with
// many splits, their ceil(k / splits)-th distances together: kMaxUm).  A
// max-heap per query in shared memory instead made every insertion a chain
// of dependent shared accesses, one query tile of 4 warps per SM and a
// separate threshold per split.  Whole calls: 10,000 queries x 1M x 128
// integers at k = 10 17.6 -> 3.7 ms (the kernel 17.3 -> 3.5 ms, 0.73 PFLOP/s),
// at k = 100 36.7 -> 7.3 ms; 777 x 99,991 x 100 floats at k = 100 2.2 - 3.3 ms
// (varying with its allocations) -> 0.44; 50 x 5,000 x 24 at k = 1 0.71 -> 0.10.
//
// A key that ties a split's own threshold has a larger id than the k kept
// (bases are visited in increasing id order) and is dropped; one that ties
// another split's threshold is kept.  A merge kernel (one warp per query)
// takes the k smallest keys over the splits.  The result -- ascending
// (distance, id), ties broken by the lower id -- depends neither on the
// split nor on the order in which thresholds are seen.
//
// A CTA takes an SM for itself: with two query tiles all 512 TMEM columns, and
// nearly all shared memory.  Beside a search on another stream, whose CTAs keep
// their queues in TMEM, it starts when those on its SM have ended; the search's
// next CTAs wait likewise.  Each kernel allocates once, holding nothing else that
// the others wait for, so these waits end.
//
// Every wait is bounded (about two seconds): a role that gives up raises the
// CTA's abort flag and the error word, the others leave their loops, copies
// still in flight and MMAs still running are waited for (again bounded), and
// the tensor memory is freed before the CTA returns.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "song_b200.h"
#include "song_kernels.cuh"

namespace song {
extern std::atomic<int64_t> g_launches;
}

namespace {

constexpr int kM = 128;            // queries per tile (MMA M, TMEM lanes)
constexpr int kN = 128;            // bases per tile (MMA N, columns of one accumulator)
constexpr int kKC = 32;            // dimensions per chunk
constexpr int kBlock = kM * kKC * 2;  // bytes of one 128 x 32 BF16 block
constexpr int kMaxStages = 8;
// A tile's norms arrive with its first stage; the copier runs at most
// kMaxStages + 2 tiles ahead of the epilogue (the MMAs of a tile wait for the
// epilogue two tiles before it).
constexpr int kNormSlots = 16;
constexpr int kMaxK = 128;
constexpr int kMaxSplits = 256;
constexpr int kSmemLimit = 232448;  // opt-in shared memory per block on sm_100
constexpr long long kWaitCycles = 4000000000LL;  // about 2 s

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N = 128, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) |
                            ((uint32_t)(kM >> 4) << 24);

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase of parity `parity`; false after ~2 s, or as soon as
// another role has raised `abort` (when given).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* abort) {
    const long long t0 = clock64();
    for (;;) {
        if (mbar_test(bar, parity)) return true;
        if (abort != nullptr && *abort) return false;
        if (clock64() - t0 > kWaitCycles) return false;
    }
}

// Shared-memory matrix descriptor (tcgen05): start, leading and stride byte
// offsets in 16-byte units, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t start, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((start >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :: "r"(tmem), "l"(ad), "l"(bd), "r"(kIdesc), "r"(acc) : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(bar) : "memory");
}

// Byte offset of element (r, k) inside one 128 x 32 block.
__host__ __device__ __forceinline__ uint32_t blk_off(int r, int k) {
    return (uint32_t)((r >> 3) * 512 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// Order-preserving map of an FP32 distance to an unsigned key (all finite
// values and +inf; -0 is folded into +0 by the caller).
__device__ __forceinline__ uint32_t ord32(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unord32(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// One side of the conversion: FP32 rows -> tiles and norms.
struct TileSide {
    const float* x;
    int64_t rows, ld, rows_pad;
    unsigned char* tiles;
    float* norm;
    int* lo_any;  // 1 when some lo value is nonzero
    bool vec;     // rows start on 16 bytes
};

// The 8 elements of row r from dimension k0 on (zero past the row or dim).
__device__ __forceinline__ void load8(const TileSide& s, int64_t r, int k0, int dim, float (&v)[8]) {
    const float* p = s.x + r * s.ld + k0;
    if (r < s.rows && s.vec && k0 + 8 <= dim) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(p));
        const float4 b = __ldg(reinterpret_cast<const float4*>(p) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = (r < s.rows && k0 + e < dim) ? __ldg(p + e) : 0.0f;
    }
}

// BF16 hi blocks of the query and base rows (padding rows and dimensions are
// zero), whether some lo value is nonzero, and the squared norms: FP64 sums
// of the FP32 squares, 32 partial sums of k = l (mod 32) added by a 16, 8, 4,
// 2, 1 butterfly, rounded to FP32 (padding rows get +inf).  One warp per 8
// rows: lane (row, group) holds 8 consecutive dimensions of each 32, so a
// warp's loads are whole 128-byte pieces of 8 rows and its stores 4 runs of
// 128 bytes; the rows are read once for both results.
__global__ void gt_tiles(const TileSide q, const TileSide b, int dim, int nch) {
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const bool isq = w < q.rows_pad / 8;
    const TileSide& s = isq ? q : b;
    const int64_t r = (isq ? w : w - q.rows_pad / 8) * 8 + (lane >> 2);
    if (r >= s.rows_pad) return;  // warp-uniform: rows_pad is a multiple of 128
    const int g = lane & 3;
    unsigned char* dst = s.tiles + (size_t)(r / kM) * 2 * nch * kBlock + blk_off((int)(r % kM), g * 8);
    double acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.0;
    bool nz = false;
    for (int c = 0; c < nch; ++c) {
        float v[8];
        load8(s, r, c * kKC + g * 8, dim, v);
        __align__(16) __nv_bfloat16 hi[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            hi[e] = __float2bfloat16_rn(v[e]);
            nz |= __bfloat162float(__float2bfloat16_rn(v[e] - __bfloat162float(hi[e]))) != 0.0f;
            acc[e] += (double)v[e] * (double)v[e];
        }
        *reinterpret_cast<uint4*>(dst + (size_t)c * kBlock) = *reinterpret_cast<const uint4*>(hi);
    }
    // partial sum l = 8 g + e: offsets 16 and 8 pair groups, 4, 2 and 1 the eight of a group
#pragma unroll
    for (int o = 2; o >= 1; o >>= 1)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1)
#pragma unroll
        for (int e = 0; e < o; ++e) acc[e] += acc[e + o];
    if (g == 0) s.norm[r] = r < s.rows ? (float)acc[0] : INFINITY;
    if (__any_sync(0xffffffffu, nz) && lane == 0) atomicOr(s.lo_any, 1);
}

// The lo blocks, of the sides that have a nonzero lo value.
__global__ void gt_lo(const TileSide q, const TileSide b, int dim, int nch) {
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const bool isq = w < q.rows_pad / 8;
    const TileSide& s = isq ? q : b;
    if (*s.lo_any == 0) return;
    const int64_t r = (isq ? w : w - q.rows_pad / 8) * 8 + (lane >> 2);
    if (r >= s.rows_pad) return;
    const int g = lane & 3;
    unsigned char* dst = s.tiles + ((size_t)(r / kM) * 2 + 1) * nch * kBlock + blk_off((int)(r % kM), g * 8);
    for (int c = 0; c < nch; ++c) {
        float v[8];
        load8(s, r, c * kKC + g * 8, dim, v);
        __align__(16) __nv_bfloat16 lo[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            lo[e] = __float2bfloat16_rn(v[e] - __bfloat162float(__float2bfloat16_rn(v[e])));
        *reinterpret_cast<uint4*>(dst + (size_t)c * kBlock) = *reinterpret_cast<const uint4*>(lo);
    }
}

struct GtArgs {
    const unsigned char* qtiles;  // [qtiles][2][nch][kBlock]
    const unsigned char* btiles;  // [btiles][2][nch][kBlock]
    const float* qnorm;           // [nq padded]
    const float* bnorm;           // [n padded]
    const int* lo;                // [0] queries, [1] bases: their lo blocks are used
    int nq, n, nch, ntiles, tiles_per_split, splits, k;
    uint32_t ring_bytes;          // shared memory of the query blocks and the stages
    unsigned long long* list;     // [nq][splits][CAP] keys, unordered
    int* count;                   // [nq][splits]
    uint32_t* bound;              // [nq] ordered bits of the smallest k-th distance of any split
    uint32_t* nth;                // [splits][nq] ordered bits of a split's um-th smallest distance
    int um, used;                 // ceil(k / used), or 0: not used; the splits that have a tile
    int* err;                     // set to 2 when a bounded wait gives up
};

// While lists of a large k fill, the splits of a query also share their um-th
// smallest distances, um = ceil(k / splits): the largest of these bounds the
// final k-th too (um of every split lie at or below it, k together), and it is
// there after the first tile, where a split's own k-th distance takes a full
// list and its cut.  A split keeps its um smallest in registers, so only for um
// <= 4: few queries, many splits (777 x 99,991 x 100 at k = 100, 36 splits,
// 0.57 -> 0.44 ms; 100 x 500,000 x 128 at k = 100 0.61 -> 0.48; 1,500 x 60,000 x
// 200 at k = 32 0.45 -> 0.41).  In instances of their own: compiled into the
// others and switched off it cost 10,000 x 1M at k = 100 23 %.
constexpr int kMaxUm = 4;

// A value t with exactly k of the valid keys (not ~0) <= t: bisection of the
// key range (keys are unique and at least k are valid).  E keys per lane.
template <int E>
__device__ __forceinline__ unsigned long long kth_bound(const unsigned long long (&key)[E], int k) {
    uint32_t mn = 0xffffffffu, mx = 0u;
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (key[e] != ~0ull) {
            mn = min(mn, (uint32_t)(key[e] >> 32));
            mx = max(mx, (uint32_t)(key[e] >> 32));
        }
    unsigned long long lo = (unsigned long long)__reduce_min_sync(0xffffffffu, mn) << 32;
    unsigned long long hi = ((unsigned long long)__reduce_max_sync(0xffffffffu, mx) << 32) | 0xfffffffeu;
    while (E > 2 && hi - lo > 3) {  // four parts per round: the three counts (at most 256) in one redux
        const unsigned long long step = (hi - lo) >> 2;
        const unsigned long long p1 = lo + step, p2 = p1 + step, p3 = p2 + step;
        unsigned c = 0;
#pragma unroll
        for (int e = 0; e < E; ++e)
            c += (key[e] <= p1 ? 1u : 0u) + (key[e] <= p2 ? 1u << 10 : 0u) + (key[e] <= p3 ? 1u << 20 : 0u);
        c = __reduce_add_sync(0xffffffffu, c);
        const unsigned c1 = c & 1023u, c2 = (c >> 10) & 1023u, c3 = c >> 20, want = (unsigned)k;
        if (c1 == want) return p1;
        if (c2 == want) return p2;
        if (c3 == want) return p3;
        if (c1 > want) hi = p1;
        else if (c2 > want) { lo = p1 + 1; hi = p2; }
        else if (c3 > want) { lo = p2 + 1; hi = p3; }
        else lo = p3 + 1;
    }
    while (lo < hi) {
        const unsigned long long mid = lo + ((hi - lo) >> 1);
        unsigned c = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) c += key[e] <= mid;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c == (unsigned)k) return mid;
        if (c > (unsigned)k) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Writes the keys <= t to out, in any order; returns how many.
template <int E>
__device__ __forceinline__ int keep_below(const unsigned long long (&key)[E], unsigned long long t,
                                          unsigned long long* out, int lane) {
    int n = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const bool in = key[e] <= t;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) out[n + __popc(m & ((1u << lane) - 1u))] = key[e];
        n += __popc(m);
    }
    return n;
}

__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
          "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
          "=r"(r[30]), "=r"(r[31])
        : "r"(addr)
        : "memory");
}

// Waits for the loads in flight; r is an operand, so no use of it moves above.
__device__ __forceinline__ void tmem_wait32(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
          "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
          "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
          "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
          "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
          "+r"(r[30]), "+r"(r[31])
        :: "memory");
}

// MT: query tiles per CTA.  CAP: list entries per query and split (a
// multiple of 32, at least k + 32, so that a chunk always fits).
template <int MT, int CAP, bool UM>
__global__ void __launch_bounds__(32 * (4 * MT + 2), 1) gt_kernel(const GtArgs a) {
    constexpr int EW = 4 * MT;  // epilogue warps
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) float bn_s[kNormSlots][kN];  // base norms of the tiles in flight
    __shared__ __align__(8) uint64_t bar_full[kMaxStages];
    __shared__ __align__(8) uint64_t bar_empty[kMaxStages];
    __shared__ __align__(8) uint64_t bar_accf[2];
    __shared__ __align__(8) uint64_t bar_acce[2];
    __shared__ __align__(8) uint64_t bar_a;
    __shared__ __align__(8) uint64_t bar_drain;
    __shared__ uint32_t tslot;
    __shared__ volatile int abort_flag;
    __shared__ int issued_s, consumed_s, a_issued_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int a_parts = a.lo[0] ? 2 : 1, b_parts = a.lo[1] ? 2 : 1;  // 1: hi only, 2: hi and lo
    // a stage carries the blocks of `group` chunks (16 to 32 KB of bases)
    const int group = min(a.nch, a_parts + b_parts == 2 ? 4 : 2), ngrp = (a.nch + group - 1) / group;
    const uint32_t b_stage = (uint32_t)(group * b_parts) * kBlock;
    // query blocks resident when they leave room for three stages of base
    // blocks, else a stage carries both
    const uint64_t a_bytes64 = (uint64_t)(MT * a_parts) * a.nch * kBlock;  // 2^32 at four million dimensions
    const bool resident = a_bytes64 + 3u * b_stage <= a.ring_bytes;
    const uint32_t a_bytes = resident ? (uint32_t)a_bytes64 : 0u;
    const uint32_t a_stage = resident ? 0u : (uint32_t)(MT * a_parts * group) * kBlock;
    const uint32_t stage_bytes = a_stage + b_stage;
    unsigned char* ring = smem + a_bytes;
    const int stages = min(kMaxStages, (int)((a.ring_bytes - a_bytes) / stage_bytes));

    const int qt = blockIdx.x, y = blockIdx.y;
    const int t_begin = y * a.tiles_per_split;
    const int t_end = min(a.ntiles, t_begin + a.tiles_per_split);
    const int ntl = max(0, t_end - t_begin);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&tslot)), "r"(2 * MT * kN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&bar_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&bar_empty[s])) : "memory");
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" :: "r"(smem_addr(&bar_accf[b])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(&bar_acce[b])), "r"(EW) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&bar_a)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&bar_drain)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_flag = 0;
        issued_s = 0;
        consumed_s = 0;
        a_issued_s = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tslot;

    if (warp == EW) {
        // ---- copier: queries once, then (tile, group) after (tile, group) around the ring ----
        if (lane == 0) {
            auto copy = [&](uint32_t dst, const unsigned char* src, uint32_t bytes, uint32_t bar) {
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                    :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
            };
            auto expect = [&](uint32_t bar, uint32_t bytes) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                             :: "r"(bar), "r"(bytes) : "memory");
            };
            const size_t part = (size_t)a.nch * kBlock;  // one part of a tile
            const unsigned char* qsrc = a.qtiles + (size_t)qt * MT * 2 * part;
            if (resident && ntl > 0) {
                const uint32_t bar = smem_addr(&bar_a);
                expect(bar, a_bytes);
                for (int mt = 0; mt < MT; ++mt)
                    copy(smem_addr(smem) + (uint32_t)(mt * a_parts) * (uint32_t)part, qsrc + mt * 2 * part,
                         (uint32_t)(a_parts * part), bar);
                a_issued_s = 1;
            }
            int s = 0, i = 0;
            uint32_t parity = 1;  // of the empty phase to wait for: the first round passes at once
            bool ok = true;
            for (int j = 0; j < ntl && ok; ++j) {
                const unsigned char* bsrc = a.btiles + (size_t)(t_begin + j) * 2 * part;
                for (int g = 0; g < ngrp; ++g) {
                    if (!mbar_wait(smem_addr(&bar_empty[s]), parity, &abort_flag)) {
                        abort_flag = 1;
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_addr(&bar_full[s]);
                    const uint32_t gb = (uint32_t)min(group, a.nch - g * group) * kBlock;  // bytes of the group, one part
                    const size_t off = (size_t)g * group * kBlock;
                    uint32_t dst = smem_addr(ring + (size_t)s * stage_bytes);
                    expect(bar, (uint32_t)(b_parts + (resident ? 0 : MT * a_parts)) * gb + (g == 0 ? kN * 4u : 0u));
                    if (!resident)
                        for (int p = 0; p < MT * a_parts; ++p, dst += (uint32_t)group * kBlock)
                            copy(dst, qsrc + ((p / a_parts) * 2 + p % a_parts) * part + off, gb, bar);
                    for (int p = 0; p < b_parts; ++p, dst += (uint32_t)group * kBlock)
                        copy(dst, bsrc + p * part + off, gb, bar);
                    if (g == 0)
                        copy(smem_addr(bn_s[j % kNormSlots]),
                             reinterpret_cast<const unsigned char*>(a.bnorm + (size_t)(t_begin + j) * kN), kN * 4u, bar);
                    ++i;
                    if (++s == stages) {
                        s = 0;
                        parity ^= 1u;
                    }
                }
            }
            issued_s = i;
        }
    } else if (warp == EW + 1) {
        // ---- MMA issuer ----
        if (lane == 0) {
            int consumed = 0, s = 0;
            uint32_t parity = 0;
            bool ok = true;
            const uint32_t ring_addr = smem_addr(ring);
            const uint64_t a_desc = umma_desc(smem_addr(smem), 128u, 512u);
            const uint64_t b_lo = (uint64_t)group * (kBlock / 16);  // from a hi block to its lo block
            const uint64_t a_lo = (uint64_t)(resident ? a.nch : group) * (kBlock / 16);
            const uint64_t a_mt = a_lo * a_parts;                   // from one query tile to the next
            if (resident && ntl > 0) ok = mbar_wait(smem_addr(&bar_a), 0u, &abort_flag);
            for (int j = 0; j < ntl && ok; ++j) {
                const int b = j & 1;
                if (j >= 2 && !mbar_wait(smem_addr(&bar_acce[b]), (uint32_t)(((j >> 1) - 1) & 1), &abort_flag)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int g = 0; g < ngrp; ++g) {
                    if (!mbar_wait(smem_addr(&bar_full[s]), parity, &abort_flag)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    // operand descriptors; a block further on adds kBlock / 16 to the address
                    // field, a K step 16.  One thread issues everything, so its instruction
                    // count per tile has to stay below the tile's tensor time: descriptors
                    // rebuilt for every product took 3,000 cycles per tile of 256 x 128 x 128.
                    const uint32_t s0 = ring_addr + (uint32_t)s * stage_bytes;
                    const uint64_t db = umma_desc(s0 + a_stage, 128u, 512u);
                    const uint64_t da = resident ? a_desc + (uint64_t)(g * group) * (kBlock / 16)
                                                 : umma_desc(s0, 128u, 512u);
                    const uint32_t acc0 = tmem + (uint32_t)(b * MT * kN);
                    const int cn = min(group, a.nch - g * group);
                    if (a_parts + b_parts == 2) {
                        for (int c = 0; c < cn; ++c) {
#pragma unroll
                            for (int ks = 0; ks < kKC / 16; ++ks) {
                                const uint64_t o = (uint64_t)(c * (kBlock / 16) + ks * 16);
#pragma unroll
                                for (int mt = 0; mt < MT; ++mt)
                                    mma_bf16(acc0 + mt * kN, da + mt * a_mt + o, db + o, (g | c | ks) ? 1u : 0u);
                            }
                        }
                    } else {
                        for (int c = 0; c < cn; ++c) {
#pragma unroll
                            for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
                                for (int ks = 0; ks < kKC / 16; ++ks) {
                                    const uint64_t o = (uint64_t)(c * (kBlock / 16) + ks * 16);
                                    const uint64_t dah = da + mt * a_mt + o, dbh = db + o;
                                    mma_bf16(acc0 + mt * kN, dah, dbh, (g | c | ks) ? 1u : 0u);
                                    if (b_parts == 2) mma_bf16(acc0 + mt * kN, dah, dbh + b_lo, 1u);
                                    if (a_parts == 2) mma_bf16(acc0 + mt * kN, dah + a_lo, dbh, 1u);
                                }
                            }
                        }
                    }
                    mma_commit(smem_addr(&bar_empty[s]));  // the stage is free once these MMAs ran
                    ++consumed;
                    if (++s == stages) {
                        s = 0;
                        parity ^= 1u;
                    }
                }
                if (ok) {
                    mma_commit(smem_addr(&bar_accf[b]));
                    // the epilogue reads the tile's norms too, which arrived on bar_full: this
                    // thread has waited for them there, and its own arrival hands that on (the
                    // commit's arrival only says that the MMAs are done)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];"
                                 :: "r"(smem_addr(&bar_accf[b])) : "memory");
                }
            }
            if (!ok) abort_flag = 1;
            consumed_s = consumed;
            // every MMA issued so far has completed before the memory goes away
            mma_commit(smem_addr(&bar_drain));
            if (!mbar_wait(smem_addr(&bar_drain), 0u, nullptr)) abort_flag = 1;
        }
    } else {
        // ---- epilogue: thread = query row = TMEM lane ----
        const int mt = warp >> 2;
        const int q = (qt * MT + mt) * kM + (warp & 3) * 32 + lane;
        const bool live = q < a.nq;
        const float qn = live ? a.qnorm[q] : 0.0f;
        unsigned long long* list = a.list + ((size_t)(live ? q : 0) * a.splits + y) * CAP;
        int cnt = 0;
        // Keys with ordered bits below `lim` enter: below this split's own k-th
        // distance, or not above another split's.  thr: |b|^2 - 2 q.b >= thr
        // implies the same of the ordered bits; NaN (every key may enter) while
        // there is no finite limit.
        uint32_t own = 0xFFFFFFFFu, lim = 0u;
        float thr = -INFINITY;
        auto set_limit = [&](uint32_t bound) {
            const uint32_t b1 = bound == 0xFFFFFFFFu ? bound : bound + 1u;
            lim = live ? min(own, b1) : 0u;
            if (live) {
                // (|q|^2 - 2 q.b) + |b|^2 in FP32 differs from |q|^2 + fma(-2, q.b,
                // |b|^2) by less than 8 units of 2^-24 of |q|^2 + |limit|
                const float d = unord32(lim);
                const float t = (d - qn) + ((fabsf(d) + qn) * (1.0f / 524288.0f) + FLT_MIN);
                // 2 q.b may overflow where |b|^2 does not only for |q|^2 above FLT_MAX / 4:
                // such a distance is -inf, which the sum without |q|^2 does not show
                thr = fabsf(t) <= FLT_MAX && qn < FLT_MAX / 8 ? t : __int_as_float(0x7fffffff);
            }
        };
        set_limit(live ? *(volatile const uint32_t*)(a.bound + q) : 0u);
        const uint32_t row = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(mt * kN);
        uint32_t seen = 0xFFFFFFFFu;  // the shared bound, read one tile before it is used
        uint32_t low[kMaxUm];         // this split's smallest distances, ascending
#pragma unroll
        for (int i = 0; i < kMaxUm; ++i) low[i] = 0xFFFFFFFFu;
        auto lowest = [&](uint32_t o) {
#pragma unroll
            for (int i = 0; i < kMaxUm; ++i) {
                const uint32_t m = min(low[i], o);
                o = max(low[i], o);
                low[i] = m;
            }
        };
        uint32_t said = 0xFFFFFFFFu;  // the last one written to a.nth
        for (int j = 0; j < ntl; ++j) {
            const int b = j & 1;
            const float* bn = bn_s[j % kNormSlots];
            if (live && (j & 3) == 3) set_limit(seen);
            if (live && (j & 3) == 2) seen = *(volatile const uint32_t*)(a.bound + q);
            if (UM && live && (j < 8 || (j & 3) == 3)) {
                const uint32_t mine = a.um == 1 ? low[0] : a.um == 2 ? low[1] : a.um == 3 ? low[2] : low[3];
                if (mine < said) *(volatile uint32_t*)(a.nth + (size_t)y * a.nq + q) = said = mine;
                uint32_t t = 0u;
#pragma unroll 8
                for (int i = 0; i < a.used; ++i) t = max(t, *(volatile const uint32_t*)(a.nth + (size_t)i * a.nq + q));
                if (t < seen) {
                    seen = min(atomicMin(a.bound + q, t), t);
                    set_limit(seen);
                }
            }
            bool ok = mbar_wait(smem_addr(&bar_accf[b]), (uint32_t)((j >> 1) & 1), &abort_flag);
            ok = __all_sync(FULL, ok);
            if (!ok) {
                abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = row + (uint32_t)(b * MT * kN);
            const int64_t col0 = (int64_t)(t_begin + j) * kN;
            uint32_t r0[32], r1[32];
            auto chunk = [&](const uint32_t (&r)[32], int c0) {
                float v[32];
                float m0 = INFINITY, m1 = INFINITY;
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const float4 n4 = *reinterpret_cast<const float4*>(bn + c0 + 4 * g);
                    v[4 * g + 0] = fmaf(-2.0f, __uint_as_float(r[4 * g + 0]), n4.x);
                    v[4 * g + 1] = fmaf(-2.0f, __uint_as_float(r[4 * g + 1]), n4.y);
                    v[4 * g + 2] = fmaf(-2.0f, __uint_as_float(r[4 * g + 2]), n4.z);
                    v[4 * g + 3] = fmaf(-2.0f, __uint_as_float(r[4 * g + 3]), n4.w);
                    m0 = fminf(fminf(m0, v[4 * g + 0]), v[4 * g + 1]);
                    m1 = fminf(fminf(m1, v[4 * g + 2]), v[4 * g + 3]);
                }
                if (!__any_sync(FULL, !(fminf(m0, m1) >= thr))) return;
                // the columns some lane of the warp may take: few of them one at a time (32
                // unrolled copies with a branch each took 7,000 cycles per chunk with one key
                // below the threshold), many of them all, without branches (one at a time is
                // 150 cycles per column: while the lists of a large k first fill, 4,800)
                unsigned mine = 0u;
#pragma unroll
                for (int jj = 0; jj < 32; ++jj) mine |= (v[jj] >= thr ? 0u : 1u) << jj;
                unsigned todo = __reduce_or_sync(FULL, mine);
                if (CAP > 64 && __popc(todo) > 8) {
                    const int64_t left = a.n - (col0 + c0);
#pragma unroll
                    for (int jj = 0; jj < 32; ++jj) {
                        const float cross2 = 2.0f * __uint_as_float(r[jj]);
                        const float d = __fadd_rn(__fadd_rn(__fsub_rn(qn, cross2), bn[c0 + jj]), 0.0f);
                        const uint32_t o = ord32(d);
                        const bool in = ((mine >> jj) & 1u) && o < lim && jj < left;
                        if (in) list[cnt] = ((unsigned long long)o << 32) | (uint32_t)(col0 + c0 + jj);
                        cnt += in;
                        if constexpr (UM) lowest(in ? o : 0xFFFFFFFFu);
                    }
                    todo = 0u;
                }
                while (todo) {
                    const int jj = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    uint32_t x;
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\t"
                        "tcgen05.wait::ld.sync.aligned;"
                        : "=r"(x) : "r"(acc + (uint32_t)(c0 + jj)) : "memory");
                    if ((mine >> jj) & 1u) {
                        const float cross2 = 2.0f * __uint_as_float(x);
                        const float d = __fadd_rn(__fadd_rn(__fsub_rn(qn, cross2), bn[c0 + jj]), 0.0f);
                        const uint32_t o = ord32(d);
                        if (o < lim && col0 + c0 + jj < a.n) {
                            list[cnt++] = ((unsigned long long)o << 32) | (uint32_t)(col0 + c0 + jj);
                            if constexpr (UM) lowest(o);
                        }
                    }
                    __syncwarp();
                }
                __syncwarp();
                unsigned full = __ballot_sync(FULL, cnt > CAP - 32);
                while (full) {  // cut the list of lane s to its k smallest keys
                    const int s = __ffs(full) - 1;
                    full &= full - 1u;
                    unsigned long long* ls = reinterpret_cast<unsigned long long*>(
                        __shfl_sync(FULL, reinterpret_cast<unsigned long long>(list), s));
                    const int n = __shfl_sync(FULL, cnt, s);
                    unsigned long long key[CAP / 32];
#pragma unroll
                    for (int e = 0; e < CAP / 32; ++e) key[e] = lane + 32 * e < n ? ls[lane + 32 * e] : ~0ull;
                    const unsigned long long kb = kth_bound(key, a.k);
                    uint32_t top = 0u;
#pragma unroll
                    for (int e = 0; e < CAP / 32; ++e)
                        if (key[e] <= kb) top = max(top, (uint32_t)(key[e] >> 32));
                    top = __reduce_max_sync(FULL, top);
                    __syncwarp();
                    keep_below(key, kb, ls, lane);
                    __syncwarp();
                    if (lane == s) {
                        cnt = a.k;
                        own = top;
                        set_limit(min(atomicMin(a.bound + q, top), top));
                    }
                }
                __syncwarp();
            };
            tmem_ld32(acc, r0);
#pragma unroll 1
            for (int c0 = 0; c0 < kN; c0 += 64) {
                tmem_wait32(r0);
                tmem_ld32(acc + (uint32_t)(c0 + 32), r1);
                chunk(r0, c0);
                tmem_wait32(r1);
                if (c0 + 64 < kN) tmem_ld32(acc + (uint32_t)(c0 + 64), r0);
                chunk(r1, c0 + 32);
            }
            // the accumulator has been read: the MMAs may overwrite it
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];"
                             :: "r"(smem_addr(&bar_acce[b])) : "memory");
        }
        if (live) a.count[(size_t)q * a.splits + y] = cnt;
    }
    __syncthreads();

    // copies still in flight when a role gave up: wait for them (bounded)
    if (abort_flag && tid == EW * 32) {
        if (a_issued_s) mbar_wait(smem_addr(&bar_a), 0u, nullptr);
        for (int i = consumed_s; i < issued_s; ++i)
            mbar_wait(smem_addr(&bar_full[i % stages]), (uint32_t)((i / stages) & 1), nullptr);
    }
    if (abort_flag && tid == 0) atomicExch(a.err, 2);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(2 * MT * kN)
                     : "memory");
}

// The k smallest keys over a query's lists, ascending; one warp per query.
// Keys above the query's shared bound cannot be among them, which leaves few
// more than k; they collect in shared memory, cut to k when it fills.
constexpr int kMergeWarps = 4, kMergeCap = 256;
__global__ void __launch_bounds__(32 * kMergeWarps) gt_merge(const unsigned long long* __restrict__ list,
                                                             const int* __restrict__ count,
                                                             const uint32_t* __restrict__ bound, int cap,
                                                             int nq, int splits, int k,
                                                             int32_t* __restrict__ ids,
                                                             float* __restrict__ dists) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int E = kMergeCap / 32;  // lists hold at most kMergeCap keys too
    __shared__ unsigned long long buf[kMergeWarps][kMergeCap];
    const int q = blockIdx.x * kMergeWarps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nq) return;
    unsigned long long* w = buf[threadIdx.x >> 5];
    unsigned long long lim = ((unsigned long long)bound[q] << 32) | 0xffffffffu;  // keys <= lim may be among the k
    int n = 0;
    unsigned long long key[E];
    auto load = [&]() {
        __syncwarp();
#pragma unroll
        for (int e = 0; e < E; ++e) key[e] = lane + 32 * e < n ? w[lane + 32 * e] : ~0ull;
        __syncwarp();
    };
    for (int s = 0; s < splits; ++s) {
        const int c = count[(size_t)q * splits + s];
        const unsigned long long* ls = list + ((size_t)q * splits + s) * cap;
        unsigned long long in_flight[E];  // the whole list at once: one round trip per split
#pragma unroll
        for (int e = 0; e < E; ++e) in_flight[e] = lane + 32 * e < c ? ls[lane + 32 * e] : ~0ull;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if (32 * e >= c) break;
            const unsigned long long x = in_flight[e];
            const bool in = x != ~0ull && x <= lim;
            const unsigned m = __ballot_sync(FULL, in);
            if (in) w[n + __popc(m & ((1u << lane) - 1u))] = x;
            n += __popc(m);
            if (n > kMergeCap - 32) {
                load();
                lim = kth_bound(key, k);
                n = keep_below(key, lim, w, lane);
                __syncwarp();
            }
        }
    }
    load();
    if (n > k) {
        n = keep_below(key, kth_bound(key, k), w, lane);
        load();
    }
    // unique keys: a key's place is the number of smaller ones
    int rank[E];
#pragma unroll
    for (int e = 0; e < E; ++e) rank[e] = 0;
    for (int i = 0; i < n; ++i) {
        const unsigned long long x = w[i];
#pragma unroll
        for (int e = 0; e < E; ++e) rank[e] += x < key[e];
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (key[e] != ~0ull) {
            ids[(size_t)q * k + rank[e]] = (int32_t)(uint32_t)(key[e] & 0xFFFFFFFFull);
            dists[(size_t)q * k + rank[e]] = unord32((uint32_t)(key[e] >> 32));
        }
    for (int i = n + lane; i < k; i += 32) {
        ids[(size_t)q * k + i] = -1;
        dists[(size_t)q * k + i] = INFINITY;
    }
}

// Splits per query tile: the count that minimises (waves of CTAs) x (tiles
// per split and its fixed cost, about kItemTiles tiles of time: start-up and
// the keys that enter before the first threshold), the smaller one on ties;
// at most 6 waves, as each split keeps a list per query.
constexpr int kItemTiles = 8;
int pick_splits(int qtiles, int ntiles, int num_sms) {
    int best = 1;
    int64_t best_cost = INT64_MAX;
    for (int s = 1; s <= std::min(kMaxSplits, ntiles); ++s) {
        const int64_t tps = (ntiles + s - 1) / s;
        const int used = (int)((ntiles + tps - 1) / tps);
        if (used != s) continue;
        const int64_t items = (int64_t)qtiles * s;
        const int64_t waves = (items + num_sms - 1) / num_sms;
        if (s > 1 && waves > 6) break;
        const int64_t cost = waves * (tps + kItemTiles);
        if (cost < best_cost) {
            best_cost = cost;
            best = s;
        }
    }
    return best;
}

}  // namespace

namespace song {

// Workspaces of calls that belong to no index come from one stream-ordered
// pool per device (safe for calls on several streams and threads at once),
// which keeps up to kPoolKeep bytes for the next call: a cudaMalloc and
// cudaFree of the workspace took 0.6 - 1.3 ms per call, most of a small
// call's time.  trim_workspaces gives the kept bytes back; destroying an
// index does, and device_alloc does before it fails (a cudaMalloc of other
// code has been seen to get them from the driver as well).
static std::mutex g_pool_mu;
static cudaMemPool_t g_pool[64] = {};
constexpr uint64_t kPoolKeep = 1ull << 30;

static cudaError_t workspace_pool(int dev, cudaMemPool_t* out) {
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (g_pool[dev] == nullptr) {
        cudaMemPoolProps pp = {};
        pp.allocType = cudaMemAllocationTypePinned;
        pp.location.type = cudaMemLocationTypeDevice;
        pp.location.id = dev;
        cudaMemPool_t p = nullptr;
        cudaError_t e = cudaMemPoolCreate(&p, &pp);
        uint64_t keep = kPoolKeep;
        if (e == cudaSuccess) e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) return e;
        g_pool[dev] = p;
    }
    *out = g_pool[dev];
    return cudaSuccess;
}

void trim_workspaces(int dev) {
    if (dev < 0 || dev >= 64) return;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (g_pool[dev] != nullptr) cudaMemPoolTrimTo(g_pool[dev], 0);
}

cudaError_t workspace_alloc(void** p, size_t bytes, cudaStream_t st) {
    int dev = 0;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = workspace_pool(dev, &pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    return e;
}

cudaError_t device_alloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) trim_workspaces(dev);
    return cudaMalloc(p, bytes);
}

// Exact kNN of device rows.  Synchronous on `st`.  err: 0 ok, 2 a wait gave up.
cudaError_t exact_knn(const float* d_base, int64_t n, int64_t ldb, int dim, const float* d_q, int nq,
                      int64_t ldq, int k, int32_t* d_ids, float* d_dists, cudaStream_t st, int* err_out) {
    *err_out = 0;
    if (nq == 0) return cudaSuccess;
    int dev = 0, num_sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const int nch = (dim + kKC - 1) / kKC;
    // two query tiles per CTA halve the base traffic per product; one where
    // padding to 256 queries would add more than a fifth to the products
    const int q1 = (nq + kM - 1) / kM, q2 = (q1 + 1) / 2;
    const int mt = 10 * q2 <= 6 * q1 ? 2 : 1;
    const int qtiles = mt == 2 ? q2 : q1, ntiles = (int)((n + kN - 1) / kN);
    const int64_t qpad = (int64_t)qtiles * mt * kM, npad = (int64_t)ntiles * kN;
    const int splits = pick_splits(qtiles, ntiles, num_sms);
    const int cap = k <= 16 ? 64 : 256;
    // one allocation, carved on 256-byte boundaries
    size_t total = 0;
    auto take = [&](size_t bytes) {
        const size_t o = total;
        total += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_q = take((size_t)qpad / kM * nch * 2 * kBlock), o_b = take((size_t)ntiles * nch * 2 * kBlock);
    const size_t o_qn = take((size_t)qpad * 4), o_bn = take((size_t)npad * 4);
    const size_t o_list = take((size_t)nq * splits * cap * 8), o_cnt = take((size_t)nq * splits * 4);
    const size_t o_flags = take(3 * sizeof(int));  // [0] query lo, [1] base lo, [2] error word
    const size_t o_bound = take((size_t)nq * 4);
    const int tps = (ntiles + splits - 1) / splits, used = (ntiles + tps - 1) / tps;
    int um = (k + used - 1) / used;
    if (cap == 64 || used == 1 || um > kMaxUm) um = 0;
    const size_t o_nth = take(um ? (size_t)nq * splits * 4 : 0);
    char* ws = nullptr;
    e = workspace_alloc(reinterpret_cast<void**>(&ws), total, st);
    if (e == cudaErrorMemoryAllocation && nq > 2 * kM) {
        // no room for the lists of all queries (512 or 2,048 bytes per query and
        // split): half of them at a time, with the same results
        cudaGetLastError();
        const int half = (nq / 2 + 2 * kM - 1) / (2 * kM) * (2 * kM);
        e = exact_knn(d_base, n, ldb, dim, d_q, half, ldq, k, d_ids, d_dists, st, err_out);
        if (e != cudaSuccess || *err_out != 0) return e;
        return exact_knn(d_base, n, ldb, dim, d_q + (int64_t)half * ldq, nq - half, ldq, k,
                         d_ids + (int64_t)half * k, d_dists + (int64_t)half * k, st, err_out);
    }
    if (e != cudaSuccess) return e;
    int* flags = reinterpret_cast<int*>(ws + o_flags);
    e = cudaMemsetAsync(flags, 0, 3 * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(ws + o_bound, 0xff, (size_t)nq * 4, st);
    if (e == cudaSuccess && um) e = cudaMemsetAsync(ws + o_nth, 0xff, (size_t)nq * splits * 4, st);
    int h_err = 0;
    if (e == cudaSuccess) {
        const auto vec = [](const float* p, int64_t ld) {
            return (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && (ld & 3) == 0;
        };
        const TileSide qs{d_q, nq, ldq, qpad, reinterpret_cast<unsigned char*>(ws + o_q),
                          reinterpret_cast<float*>(ws + o_qn), flags, vec(d_q, ldq)};
        const TileSide bs{d_base, n, ldb, npad, reinterpret_cast<unsigned char*>(ws + o_b),
                          reinterpret_cast<float*>(ws + o_bn), flags + 1, vec(d_base, ldb)};
        const unsigned blocks = (unsigned)((qpad + npad) / 8 + 7) / 8;
        gt_tiles<<<blocks, 256, 0, st>>>(qs, bs, dim, nch);
        gt_lo<<<blocks, 256, 0, st>>>(qs, bs, dim, nch);
        GtArgs a;
        a.qtiles = qs.tiles;
        a.btiles = bs.tiles;
        a.qnorm = qs.norm;
        a.bnorm = bs.norm;
        a.lo = flags;
        a.nq = nq;
        a.n = (int)n;
        a.nch = nch;
        a.ntiles = ntiles;
        a.tiles_per_split = tps;
        a.splits = splits;
        a.k = k;
        a.list = reinterpret_cast<unsigned long long*>(ws + o_list);
        a.count = reinterpret_cast<int*>(ws + o_cnt);
        a.bound = reinterpret_cast<uint32_t*>(ws + o_bound);
        a.nth = reinterpret_cast<uint32_t*>(ws + o_nth);
        a.um = um;
        a.used = used;
        a.err = flags + 2;
        void (*kern)(const GtArgs) = mt == 2 ? gt_kernel<2, 64, false> : gt_kernel<1, 64, false>;
        if (cap == 256) {
            kern = mt == 2 ? gt_kernel<2, 256, false> : gt_kernel<1, 256, false>;
            if (um) kern = mt == 2 ? gt_kernel<2, 256, true> : gt_kernel<1, 256, true>;
        }
        cudaFuncAttributes fa;
        e = cudaFuncGetAttributes(&fa, kern);
        if (e == cudaSuccess) {
            a.ring_bytes = (uint32_t)((kSmemLimit - (int)fa.sharedSizeBytes) / 1024 * 1024);
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a.ring_bytes);
        }
        if (e == cudaSuccess) {
            kern<<<dim3((unsigned)qtiles, (unsigned)splits), 32 * (4 * mt + 2), a.ring_bytes, st>>>(a);
            gt_merge<<<(unsigned)((nq + kMergeWarps - 1) / kMergeWarps), 32 * kMergeWarps, 0, st>>>(
                a.list, a.count, a.bound, cap, nq, splits, k, d_ids, d_dists);
            g_launches.fetch_add(4, std::memory_order_relaxed);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_err, flags + 2, sizeof(int), cudaMemcpyDeviceToHost, st);
    // freed ahead of the synchronisation: a free that is still on its way keeps
    // the memory from every other allocation until the stream is next waited for
    const cudaError_t ef = cudaFreeAsync(ws, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    *err_out = h_err;
    return e != cudaSuccess ? e : ef;
}

}  // namespace song

extern "C" {

song_status song_exact_knn_device(const float* d_base, int64_t n, int64_t ldb, int dim,
                                  const float* d_queries, int nq, int64_t ldq, int k,
                                  int32_t* d_ids, float* d_dists, void* stream) {
    if (dim < 1) return song::set_error(SONG_ERR_INVALID_ARG, "dim must be >= 1");
    if (n < 1 || n > (int64_t)INT32_MAX - kN) return song::set_error(SONG_ERR_INVALID_ARG, "n out of range");
    if (nq < 0) return song::set_error(SONG_ERR_INVALID_ARG, "nq must be >= 0");
    if (k < 1 || k > kMaxK) return song::set_error(SONG_ERR_INVALID_ARG, "k must be in [1, 128]");
    if (ldb < dim || ldq < dim) return song::set_error(SONG_ERR_INVALID_ARG, "ldb and ldq must be >= dim");
    if (nq > 0 && (d_base == nullptr || d_queries == nullptr || d_ids == nullptr || d_dists == nullptr))
        return song::set_error(SONG_ERR_INVALID_ARG, "base, queries, ids or dists is NULL");
    int err = 0;
    const cudaError_t e = song::exact_knn(d_base, n, ldb, dim, d_queries, nq, ldq, k, d_ids, d_dists,
                                          (cudaStream_t)stream, &err);
    if (e != cudaSuccess) {
        char buf[160];
        std::snprintf(buf, sizeof(buf), "exact kNN: %s", cudaGetErrorString(e));
        return song::set_error(SONG_ERR_CUDA, buf);
    }
    if (err != 0) return song::set_error(SONG_ERR_TIMEOUT, "exact kNN: a bounded wait gave up");
    return SONG_OK;
}

song_status song_exact_knn(const float* base, int64_t n, int dim, const float* queries, int nq, int k,
                           int32_t* ids, float* dists) {
    if (nq == 0) return SONG_OK;
    if (base == nullptr || queries == nullptr || ids == nullptr || dists == nullptr)
        return song::set_error(SONG_ERR_INVALID_ARG, "base, queries, ids or dists is NULL");
    if (dim < 1 || n < 1 || nq < 0) return song::set_error(SONG_ERR_INVALID_ARG, "bad shape");
    float *d_b = nullptr, *d_q = nullptr, *d_d = nullptr;
    int32_t* d_i = nullptr;
    cudaStream_t st = nullptr;
    const size_t bb = (size_t)n * dim * 4, qb = (size_t)nq * dim * 4, ob = (size_t)nq * k;
    cudaError_t e = song::device_alloc((void**)&d_b, bb);
    if (e == cudaSuccess) e = song::device_alloc((void**)&d_q, qb);
    if (e == cudaSuccess) e = song::device_alloc((void**)&d_i, ob * 4);
    if (e == cudaSuccess) e = song::device_alloc((void**)&d_d, ob * 4);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_b, base, bb, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_q, queries, qb, cudaMemcpyHostToDevice, st);
    song_status s = SONG_OK;
    if (e == cudaSuccess) {
        s = song_exact_knn_device(d_b, n, dim, dim, d_q, nq, dim, k, d_i, d_d, st);
        if (s == SONG_OK) {
            e = cudaMemcpyAsync(ids, d_i, ob * 4, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(dists, d_d, ob * 4, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        }
    }
    cudaFree(d_b);
    cudaFree(d_q);
    cudaFree(d_i);
    cudaFree(d_d);
    if (st) cudaStreamDestroy(st);
    if (s != SONG_OK) return s;
    if (e != cudaSuccess) {
        char buf[160];
        std::snprintf(buf, sizeof(buf), "exact kNN: %s", cudaGetErrorString(e));
        return song::set_error(SONG_ERR_CUDA, buf);
    }
    return SONG_OK;
}

}  // extern "C"

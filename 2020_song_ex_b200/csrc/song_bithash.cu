// song_bithash.cu -- sign-random-projection codes (BitHash) on the GPU.
//
// The reference projects every base vector and every query on one CPU
// thread (BitHash::project / project_all, bitHash.h:32-56): bit b of word w
// is set when the FP32 dot product of hyperplane R[w*32+b] with the vector is
// > 0, the dot being summed in increasing d as `dot += R[row*dim+d] * x[d]`.
// The reference is built with plain -O3 for x86-64, so each step is an FP32
// multiply rounded to nearest, then an FP32 add rounded to nearest (no fused
// multiply-add).  This kernel performs exactly those two roundings per step
// (__fmul_rn, __fadd_rn: never contracted) in the same d order, so every
// code is bit-identical to the reference's, including the signs of dot
// products that land near zero.
//
// Only the sign of that sum is wanted, so the tensor cores decide most bits
// and the sequential sum only those near zero.  x = xh + xl and r = rh + rl
// are split into BF16 parts; xh.rh and xh.rl + xl.rh are accumulated in two
// FP32 accumulators, and their sum m differs from the reference's sum by less
// than error_factor(dim) * |x| |r| (see there).  A bit with |m| above that
// bound has the sign of m; the others (about one in 1,300 at 256 dimensions
// of Gaussian data) are summed as above.  Every comparison with a NaN, an
// overflow or a norm near the underflow range counts as "near zero", and if a
// bounded wait gives up the CTA sums all of its remaining bits that way.  The
// norms are each vector's and each hyperplane's own: one that has no bound
// sends its own bits to the sums and no others.
//
// One CTA takes 128 hyperplanes (4 code words), their BF16 parts resident in
// shared memory up to 288 dimensions, and walks over tiles of 128 vectors;
// the CTAs of the other words walk the same tiles at the same time, so x is
// read from HBM once.  Warps have fixed roles:
//   8 converters load chunks of 128 vectors x 32 dimensions (two chunks
//     ahead in registers), split them into the tensor cores' operand layout in a
//     ring of stages, and sum the squares for the bound;
//   1 thread issues tcgen05.mma kind::f16 (M = N = 128, K = 16);
//   2 sets of 4 epilogue warps, one per accumulator buffer, turn signs into
//     code words with two funnel shifts per bit, free the buffer and then sum
//     the near-zero bits of their tile, one per lane, under the next tile's
//     products.
// Two buffers of two accumulators are all 512 TMEM columns: beside a search on
// another stream, whose CTAs keep their queues in TMEM, a CTA starts when those
// on its SM have ended (it needs the SM's shared memory and registers too), and
// the search's next ones wait for it.  Neither allocates twice: the waits end.
// A tile where a warp finds more than kDense such bits is marked and summed
// whole by all warps at the end (sum_left), as all tiles are above kTensorDim
// dimensions.  So the time does not hang on the data: 100,000 x 256 -> 512 bits
// 0.17 ms, with a zero hyperplane 0.17, a tiny one 0.28, one tiny vector in 32
// 0.64, all vectors tiny 1.29 (the sums of all bits by a kernel made for them
// 1.35; with the largest norm for all 128 hyperplanes and each lane summing its
// own vector's bits 14.0, 14.0, 5.3 and 14.0 ms).
// The floor is 3 products per multiply of the projection on the tensor cores
// (0.14 ms for 290,000 x 256 -> 512 bits) or one pass over x (0.05 ms).  The
// sums of all bits on the CUDA cores, 255 registers per thread and 8 warps per
// SM, took 3.81 ms; this takes 0.41 ms.  What bounds it is the converters' loads
// of x (in a form that took 0.47 ms: without products 0.41, without near-zero
// sums 0.43).
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "song_b200.h"
#include "song_kernels.cuh"

namespace song {
extern std::atomic<int64_t> g_launches;
}

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kTV = 128;              // vectors per tile (MMA M, TMEM lanes)
constexpr int kTB = 128;              // hyperplanes per CTA (MMA N)
constexpr int kWords = kTB / 32;      // code words per CTA
constexpr int kDC = 32;               // dimensions per chunk
constexpr int kBlock = 128 * kDC * 2; // bytes of one 128 x 32 BF16 block
constexpr int kResChunks = 9;         // resident hyperplanes: at most 9 chunks (288 dimensions)
constexpr int kStagesRes = 4, kStagesStream = 6;
constexpr int kThrSlots = 8;          // the converters run at most 8 tiles ahead of the epilogue: the
                                      // ring's chunks and 2 tiles in the accumulators
constexpr int kEpi = 8, kConv = 8;    // epilogue and converter warps
constexpr int kThreads = 32 * (kEpi + 1 + kConv);
constexpr int kItems = 128;           // near-zero bits a warp collects before it sums them
// With more near-zero bits among a warp's 4,096 the whole tile is summed at the
// end: 32 of them take about 16,000 cycles here (dependent loads and sums), the
// tile 80,000 there, by all warps.
constexpr int kDense = 256;
// The bound grows with the dimension and the sums' spread against it shrinks: 4 %
// of the bits are near zero at 4,096 dimensions (10,000 vectors -> 256 bits 1.59
// ms, 1.92 by a kernel of sequential sums) and 7 % at 6,000, where most tiles
// would be summed whole after the products (4.9 ms; 2.6 without them).
constexpr int kTensorDim = 4096;
constexpr int kSeqBits = 1024;        // marks of such tiles (each for a run of tiles when there are more)
constexpr float kMinNorm2 = 1e-24f;   // smaller squared norms have no bound: products of two such vectors
                                      // stay far above what underflow can take away (2^-126 a product)
constexpr long long kWaitCycles = 4000000000LL;  // about 2 s

// Bound on |m - s| / (|x| |r|), with S = sum |x_i r_i| <= |x| |r|, u = 2^-24:
//  * x - xh - xl is at most 2^-18 |x| (two roundings to 8 bits), so the
//    products left out, xl.rl and the two remainders, are below 3.1 * 2^-18 S;
//  * each tcgen05.mma adds 16 exact products and the accumulator, every one
//    of them off by at most 2^-23 of the largest when they are aligned: 17 *
//    2^-23 S per instruction, dim / 16 of them for xh.rh; the other
//    accumulator holds terms 2^-8 as large (twice as many instructions).  How
//    far it rounds is an assumption, no document says: sums made to lose most
//    (a large part taken back) and 5 million Gaussian ones still had every sign
//    right with an eighth of this bound, and not with a 64th;
//  * the reference's sum itself: dim products and sums, below (dim + 1) u S,
//    and the final m = main + cross below 2 u S.
// The norms are FP32 sums of squares: 2^-10 covers their rounding.
__host__ __device__ inline float error_factor(int dim) {
    const float steps = (float)((dim + 15) / 16);
    return (3.1f / 262144.0f + steps * (17.0f / 8388608.0f) * (1.0f + 2.0f / 256.0f) +
            ((float)dim + 4.0f) / 16777216.0f) * (1.0f + 1.0f / 1024.0f);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Waits for the phase of parity `parity`; false after about 2 s, or as soon
// as another warp has given up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if (*abort) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abort = 1;
            return false;
        }
    }
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_addr(bar)) : "memory");
}

// Shared-memory matrix descriptor (tcgen05): start, leading and stride byte
// offsets in 16-byte units, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t start) {
    return (uint64_t)((start >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) |
           ((uint64_t)(512u >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N = 128, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTB >> 3) << 17) |
                            ((uint32_t)(kTV >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :: "r"(tmem), "l"(ad), "l"(bd), "r"(kIdesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait16(uint32_t (&a)[16], uint32_t (&b)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]),
          "+r"(a[7]), "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]),
          "+r"(a[14]), "+r"(a[15])
        :: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(b[i]));
}

// 128 rows of FP32: the vectors of a tile or the hyperplanes of a CTA.
struct Rows {
    const float* p;   // row 0
    int64_t ld;
    int64_t count;    // rows that exist; the others read as zero
    int dim;
    bool vec;         // rows start on 16 bytes
};

// This lane's 8 elements of a chunk of 8 rows x 32 dimensions: row
// (lane >> 1) & 7, dimensions 4 (lane & 1) + 8 (lane >> 4) + 16 h + 0 .. 3 for
// h = 0, 1 (zero past the last row and dimension).  A load then takes whole
// 32-byte sectors and a store to the operand layout 128 bytes of banks in a
// row; with 4 lanes per row side by side 70 % of the shared-memory accesses
// were bank conflicts and every sector was fetched twice.
__device__ __forceinline__ int lane_row(int lane) { return (lane >> 1) & 7; }
__device__ __forceinline__ int lane_dim(int lane) { return 4 * (lane & 1) + 8 * (lane >> 4); }
__device__ __forceinline__ void load8(const Rows& s, int64_t r, int k0, float (&v)[8]) {
    const float* p = s.p + r * s.ld + k0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (r < s.count && s.vec && k0 + 16 * h + 4 <= s.dim) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(p + 16 * h));
            v[4 * h + 0] = a.x;
            v[4 * h + 1] = a.y;
            v[4 * h + 2] = a.z;
            v[4 * h + 3] = a.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                v[4 * h + e] = (r < s.count && k0 + 16 * h + e < s.dim) ? __ldg(p + 16 * h + e) : 0.0f;
        }
    }
}

// Their BF16 hi and lo parts into the operand blocks at hi and hi + lo_off
// (r8: group of 8 rows): K-major, no swizzle, 8 x 16-byte core matrices 128 B
// apart along K, groups of 8 rows 512 B apart.
__device__ __forceinline__ void store_split(unsigned char* hi, uint32_t lo_off, int r8, int lane, const float (&v)[8]) {
    unsigned char* o = hi + r8 * 512 + (lane >> 4) * 128 + lane_row(lane) * 16 + (lane & 1) * 8;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        __align__(8) __nv_bfloat162 a[2], b[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float x = v[4 * h + 2 * e], y = v[4 * h + 2 * e + 1];
            a[e] = __floats2bfloat162_rn(x, y);
            const float2 f = __bfloat1622float2(a[e]);
            b[e] = __floats2bfloat162_rn(x - f.x, y - f.y);
        }
        *reinterpret_cast<uint2*>(o + h * 256) = *reinterpret_cast<const uint2*>(a);
        *reinterpret_cast<uint2*>(o + h * 256 + lo_off) = *reinterpret_cast<const uint2*>(b);
    }
}

// The reference's sum: a rounded product, then a rounded sum, in increasing d.
__device__ __noinline__ float dot_seq(const float* __restrict__ r, const float* __restrict__ x, int dim, bool vec) {
    float s = 0.0f;
    int d = 0;
    if (vec) {
#pragma unroll 8
        for (; d + 4 <= dim; d += 4) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(r + d));
            const float4 b = __ldg(reinterpret_cast<const float4*>(x + d));
            s = __fadd_rn(s, __fmul_rn(a.x, b.x));
            s = __fadd_rn(s, __fmul_rn(a.y, b.y));
            s = __fadd_rn(s, __fmul_rn(a.z, b.z));
            s = __fadd_rn(s, __fmul_rn(a.w, b.w));
        }
    }
#pragma unroll 4
    for (; d < dim; ++d) s = __fadd_rn(s, __fmul_rn(__ldg(r + d), __ldg(x + d)));
    return s;
}

struct BhArgs {
    Rows R;           // all hyperplanes
    Rows x;           // all vectors
    uint32_t* codes;
    int64_t ldc;
    int words;        // code words per vector
    int groups;       // CTAs side by side: ceil(words / kWords)
    int per_group;    // CTAs of one group of words
    int tv;           // vectors per tile: kTV, or (without tensor) a half or a quarter of it
    int64_t tiles;    // tiles of tv vectors
    int nch;
    float factor;     // error_factor(dim)
    bool tensor;      // signs from the tensor cores (dim <= kTensorDim)
};

// What sum_left needs, in shared memory: nothing of it is kept in registers
// through the kernel's main loops.
struct Left {
    BhArgs a;
    int64_t tiles, first;             // this CTA's tiles: first + i * a.per_group
    int group, shift;                 // mark of tile i: i >> shift
    uint32_t marks[kSeqBits / 32];
};

// All bits of the marked tiles by the reference's sums, the whole CTA: 16 warps
// of 32 vectors x 32 hyperplanes, a lane 4 x 8 of them (12 values from shared
// memory for 32 products; with 32 hyperplanes per lane the loads took twice the
// time of the sums).  Chunks of 32 dimensions go through shared memory
// transposed, the next one in flight in registers.
__device__ __noinline__ void sum_left(const Left& l, float* sh) {
    constexpr int kPer = kTV * kDC / 512;  // elements per thread and side
    constexpr int kPad = 128 + 4;
    float *xs = sh, *rs = sh + kDC * kPad;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int vb = (warp >> 2) * 32 + 4 * (lane >> 2), hb = (warp & 3) * 32 + 8 * (lane & 3);
    const int dim = l.a.R.dim, nr = (int)min((int64_t)kTB, l.a.R.count - (int64_t)l.group * kTB);
    const bool mine = t < 512 && (warp & 3) * 32 < nr && (warp >> 2) * 32 < l.a.tv;
    const float* R = l.a.R.p + (int64_t)(l.group * kTB + warp) * l.a.R.ld + lane;
    for (int64_t i = 0; i < l.tiles; ++i) {
        const int m = (int)(i >> l.shift);
        if (!((l.marks[m >> 5] >> (m & 31)) & 1u)) continue;
        const int64_t v0 = (l.first + i * l.a.per_group) * l.a.tv;
        const float* x = l.a.x.p + (v0 + warp) * l.a.x.ld + lane;
        const int nx = (int)min((int64_t)l.a.tv, l.a.x.count - v0);
        float px[kPer], pr[kPer];
        auto fetch = [&](int d0) {
            const bool in = t < 512 && d0 + lane < dim;
#pragma unroll
            for (int e = 0; e < kPer; ++e) {
                px[e] = in && e * 16 + warp < nx ? __ldg(x + e * 16 * l.a.x.ld + d0) : 0.0f;
                pr[e] = in && e * 16 + warp < nr ? __ldg(R + e * 16 * l.a.R.ld + d0) : 0.0f;
            }
        };
        float s[4][8];
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int j = 0; j < 8; ++j) s[p][j] = 0.0f;
        fetch(0);
        for (int d0 = 0; d0 < dim; d0 += kDC) {
            __syncthreads();  // the chunk before has been read
            if (t < 512) {
#pragma unroll
                for (int e = 0; e < kPer; ++e) {
                    xs[lane * kPad + e * 16 + warp] = px[e];
                    rs[lane * kPad + e * 16 + warp] = pr[e];
                }
            }
            __syncthreads();
            if (d0 + kDC < dim) fetch(d0 + kDC);
            if (!mine) continue;
            const int cl = min(kDC, dim - d0);
#pragma unroll 2
            for (int d = 0; d < cl; ++d) {
                const float4 x4 = *reinterpret_cast<const float4*>(xs + d * kPad + vb);
                const float4 ra = *reinterpret_cast<const float4*>(rs + d * kPad + hb);
                const float4 rb = *reinterpret_cast<const float4*>(rs + d * kPad + hb + 4);
                const float xv[4] = {x4.x, x4.y, x4.z, x4.w};
                const float rv[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int j = 0; j < 8; ++j) s[p][j] = __fadd_rn(s[p][j], __fmul_rn(rv[j], xv[p]));
            }
        }
        uint32_t* codes = l.a.codes + v0 * l.a.ldc + l.group * kWords + (warp & 3);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            uint32_t bits = 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j) bits |= (s[p][j] > 0.0f ? 1u : 0u) << j;
            bits <<= 8 * (lane & 3);
            bits |= __shfl_xor_sync(FULL, bits, 1);
            bits |= __shfl_xor_sync(FULL, bits, 2);
            if (mine && (lane & 3) == p && vb + p < nx) codes[(vb + p) * l.a.ldc] = bits;
        }
    }
}

template <bool RES>
__global__ void __launch_bounds__(kThreads, 1) bithash_kernel(const BhArgs a) {
    constexpr int kStages = RES ? kStagesRes : kStagesStream;
    constexpr uint32_t kStageBytes = (RES ? 2 : 4) * kBlock;  // xh, xl (, rh, rl)
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar_full[kStages], bar_empty[kStages], bar_accf[2], bar_acce[2], bar_drain;
    __shared__ float thr_s[kThrSlots][kTV];  // |x| of the vectors of the tiles in flight
    __shared__ uint16_t item_s[kEpi][kItems];
    __shared__ uint32_t fix_s[kEpi][32 * kWords];
    __shared__ Left left_s;
    __shared__ uint32_t tslot;
    __shared__ __align__(16) float rn_s[kTB];  // error_factor * |r| of each hyperplane
    __shared__ volatile int abort_flag, never;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char* r_blocks = smem;                                       // RES: [hi, lo][nch][kBlock]
    unsigned char* ring = smem + (RES ? (size_t)2 * a.nch * kBlock : 0);
    const uint32_t r_lo = (uint32_t)a.nch * kBlock;

    const int group = blockIdx.x % a.groups;
    const int64_t first = blockIdx.x / a.groups;
    int64_t mytiles = first < a.tiles ? (a.tiles - first + a.per_group - 1) / a.per_group : 0;
    if (tid < kSeqBits / 32) left_s.marks[tid] = a.tensor ? 0u : FULL;
    if (tid == 0) {
        left_s.a = a;
        left_s.tiles = mytiles;
        left_s.first = first;
        left_s.group = group;
        left_s.shift = 0;
        while ((mytiles >> left_s.shift) >= kSeqBits) ++left_s.shift;
    }
    if (!a.tensor) mytiles = 0;  // all tiles are left over
    Rows R = a.R;
    R.p += (int64_t)group * kTB * R.ld;
    R.count = min((int64_t)kTB, R.count - (int64_t)group * kTB);

    if (a.tensor && warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&tslot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&bar_full[s], kConv);
            mbar_init(&bar_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bar_accf[b], 2);
            mbar_init(&bar_acce[b], 4);
        }
        mbar_init(&bar_drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_flag = 0;
        never = 0;
    }
    __syncthreads();
    // the hyperplanes' norms and (RES) operand blocks: a warp per 8 of them.  A
    // hyperplane without a bound (norm not finite or near underflow) has all its
    // bits summed (+inf); one of zeros has all clear whatever the vector (-inf:
    // the bound is below every |m|, and m is 0)
    const int kd = lane_dim(lane);
    for (int r8 = a.tensor ? warp : kTB; r8 < kTB / 8; r8 += kThreads / 32) {
        const int r = r8 * 8 + lane_row(lane);
        float q = 0.0f;
        unsigned any = 0u;
        for (int c = 0; c < a.nch; ++c) {
            float v[8];
            load8(R, r, c * kDC + kd, v);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                q = fmaf(v[e], v[e], q);
                any |= __float_as_uint(v[e]) << 1;
            }
            if constexpr (RES) store_split(r_blocks + (size_t)c * kBlock, r_lo, r8, lane, v);
        }
#pragma unroll
        for (int o = 1; o <= 16; o <<= 4) {
            q += __shfl_xor_sync(FULL, q, o);
            any |= __shfl_xor_sync(FULL, any, o);
        }
        if ((lane & 17) == 0) rn_s[r] = any == 0u ? -INFINITY : (q >= kMinNorm2 ? a.factor * sqrtf(q) : INFINITY);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tslot;

    if (warp > kEpi) {
        // ---- converters ----
        const int w = warp - kEpi - 1;
        constexpr int kT = RES ? 2 : 4;  // 8 vectors each, then (streamed) 8 hyperplanes each
        const int r0 = w * 8 + lane_row(lane);
        const int64_t total = mytiles * a.nch;
        int64_t fv0 = first * kTV;  // next chunk to load: first vector of its tile, chunk
        int fc = 0;
        auto fetch = [&](float (&d)[kT][8]) {
            load8(a.x, fv0 + r0, fc * kDC + kd, d[0]);
            load8(a.x, fv0 + r0 + 64, fc * kDC + kd, d[1]);
            if constexpr (!RES) {
                load8(R, r0, fc * kDC + kd, d[2]);
                load8(R, r0 + 64, fc * kDC + kd, d[3]);
            }
            if (++fc == a.nch) {
                fc = 0;
                fv0 += (int64_t)a.per_group * kTV;
            }
        };
        int s = 0, c = 0, slot = 0;
        uint32_t parity = 1;  // the first round of the ring passes at once
        float q0 = 0.0f, q1 = 0.0f;
        unsigned any0 = 0u, any1 = 0u;
        auto chunk = [&](float (&v)[kT][8], bool more) {
            if (!__all_sync(FULL, mbar_wait(smem_addr(&bar_empty[s]), parity, &abort_flag))) return false;
            unsigned char* st = ring + (size_t)s * kStageBytes;
            store_split(st, kBlock, w, lane, v[0]);
            store_split(st, kBlock, w + 8, lane, v[1]);
            if constexpr (!RES) {
                store_split(st + 2 * kBlock, kBlock, w, lane, v[2]);
                store_split(st + 2 * kBlock, kBlock, w + 8, lane, v[3]);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                q0 = fmaf(v[0][e], v[0][e], q0);
                q1 = fmaf(v[1][e], v[1][e], q1);
                any0 |= __float_as_uint(v[0][e]) << 1;
                any1 |= __float_as_uint(v[1][e]) << 1;
            }
            if (more) fetch(v);
            if (++c == a.nch) {
                c = 0;
#pragma unroll
                for (int o = 1; o <= 16; o <<= 4) {
                    q0 += __shfl_xor_sync(FULL, q0, o);
                    q1 += __shfl_xor_sync(FULL, q1, o);
                    any0 |= __shfl_xor_sync(FULL, any0, o);
                    any1 |= __shfl_xor_sync(FULL, any1, o);
                }
                // a zero vector's sums are zero (every bit certain: 0 > -1, clear); a norm
                // near underflow, as one that is not finite, has no bound
                if ((lane & 17) == 0) {
                    thr_s[slot][r0] = any0 == 0u ? -1.0f : (q0 >= kMinNorm2 ? sqrtf(q0) : INFINITY);
                    thr_s[slot][r0 + 64] = any1 == 0u ? -1.0f : (q1 >= kMinNorm2 ? sqrtf(q1) : INFINITY);
                }
                slot = (slot + 1) % kThrSlots;
                q0 = q1 = 0.0f;
                any0 = any1 = 0u;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_full[s]);
            if (++s == kStages) {
                s = 0;
                parity ^= 1u;
            }
            return true;
        };
        float va[kT][8], vb[kT][8];  // the next two chunks
        if (total > 0) fetch(va);
        if (total > 1) fetch(vb);
        for (int64_t k = 0; k < total; k += 2) {
            if (!chunk(va, k + 2 < total)) break;
            if (k + 1 < total && !chunk(vb, k + 3 < total)) break;
        }
    } else if (warp == kEpi) {
        // ---- MMA issuer ----
        if (lane == 0) {
            int s = 0;
            uint32_t parity = 0;
            bool ok = true;
            const uint32_t ring_addr = smem_addr(ring);
            const uint64_t r_desc = umma_desc(smem_addr(r_blocks));
            for (int64_t i = 0; i < mytiles && ok; ++i) {
                const int b = (int)(i & 1);
                if (i >= 2 && !mbar_wait(smem_addr(&bar_acce[b]), (uint32_t)(((i >> 1) - 1) & 1), &abort_flag)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t main = tmem + (uint32_t)(b * 2 * kTB), cross = main + kTB;
                for (int c = 0; c < a.nch; ++c) {
                    ok = mbar_wait(smem_addr(&bar_full[s]), parity, &abort_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t xh = umma_desc(ring_addr + (uint32_t)s * kStageBytes), xl = xh + kBlock / 16;
                    const uint64_t rh = RES ? r_desc + (uint64_t)(c * (kBlock / 16)) : xl + kBlock / 16;
                    const uint64_t rl = RES ? rh + r_lo / 16 : rh + kBlock / 16;
#pragma unroll
                    for (int ks = 0; ks < kDC / 16; ++ks) {
                        const uint32_t acc = (c | ks) ? 1u : 0u;
                        mma_bf16(main, xh + ks * 16, rh + ks * 16, acc);
                        mma_bf16(cross, xh + ks * 16, rl + ks * 16, acc);
                        mma_bf16(cross, xl + ks * 16, rh + ks * 16, 1u);
                    }
                    mma_commit(&bar_empty[s]);  // the stage is free once these MMAs ran
                    if (++s == kStages) {
                        s = 0;
                        parity ^= 1u;
                    }
                }
                if (ok) {
                    mma_commit(&bar_accf[b]);
                    // the epilogue reads the tile's bounds (thr_s) too, which arrived on bar_full:
                    // this thread has waited there, and its own arrival hands that on (the
                    // commit's arrival only says that the MMAs are done)
                    mbar_arrive(&bar_accf[b]);
                }
            }
            // every MMA issued has completed before the memory goes away
            if (a.tensor) {
                mma_commit(&bar_drain);
                mbar_wait(smem_addr(&bar_drain), 0u, &never);
            }
        }
    } else {
        // ---- epilogue: set b reads accumulator buffer b; thread = vector = TMEM lane ----
        const int b = warp >> 2;
        const int row = (warp & 3) * 32 + lane;
        const uint32_t acc = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(b * 2 * kTB);
        const bool vec = a.x.vec && a.R.vec;
        bool ok = true;
        for (int64_t i = b; i < mytiles; i += 2) {
            const int64_t v0 = (first + i * a.per_group) * kTV;
            const int64_t v = v0 + row;
            uint32_t word[kWords], unc[kWords];
            if (ok) ok = __all_sync(FULL, mbar_wait(smem_addr(&bar_accf[b]), (uint32_t)((i >> 1) & 1), &abort_flag));
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const float thr = thr_s[i % kThrSlots][row];
#pragma unroll
                for (int w = 0; w < kWords; ++w) {
                    uint32_t bits = 0u, sure = 0u;
#pragma unroll
                    for (int h = 1; h >= 0; --h) {
                        uint32_t m[16], x[16];
                        tmem_ld16(acc + (uint32_t)(w * 32 + h * 16), m);
                        tmem_ld16(acc + (uint32_t)(kTB + w * 32 + h * 16), x);
                        tmem_wait16(m, x);
#pragma unroll
                        for (int j4 = 3; j4 >= 0; --j4) {
                            const float4 rn4 = *reinterpret_cast<const float4*>(rn_s + w * 32 + h * 16 + 4 * j4);
                            const float rn[4] = {rn4.x, rn4.y, rn4.z, rn4.w};
#pragma unroll
                            for (int e = 3; e >= 0; --e) {  // sign of 0 - sum, sign of bound - |sum|
                                const int j = 4 * j4 + e;
                                const float sum = __fadd_rn(__uint_as_float(m[j]), __uint_as_float(x[j]));
                                bits = __funnelshift_l(__float_as_uint(__fsub_rn(0.0f, sum)), bits, 1);
                                sure = __funnelshift_l(__float_as_uint(fmaf(thr, rn[e], -fabsf(sum))), sure, 1);
                            }
                        }
                    }
                    word[w] = bits;
                    unc[w] = ~sure;
                }
                // the accumulator has been read: the MMAs may overwrite it
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_acce[b]);
            } else {
#pragma unroll
                for (int w = 0; w < kWords; ++w) {
                    word[w] = 0u;
                    unc[w] = FULL;
                }
            }
            const int nw = min(kWords, a.words - group * kWords);
            int cnt = 0;
#pragma unroll
            for (int w = 0; w < kWords; ++w) {
                if (v >= a.x.count || w >= nw) unc[w] = 0u;
                cnt += __popc(unc[w]);
            }
            int before = cnt;  // inclusive prefix over the lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, before, o);
                if (lane >= o) before += t;
            }
            const int total = __shfl_sync(FULL, before, 31);
            before -= cnt;
            if (total > kDense) {  // many (vectors without a bound, or so many dimensions that it is wide)
                const int m = (int)(i >> left_s.shift);
                if (lane == 0) atomicOr(&left_s.marks[m >> 5], 1u << (m & 31));
                continue;
            } else if (total > 0) {  // few: spread over the lanes, kItems at a time
#pragma unroll
                for (int w = 0; w < kWords; ++w) fix_s[warp][lane * kWords + w] = word[w] & ~unc[w];
                for (int done = 0; done < total; done += kItems) {
#pragma unroll
                    for (int w = 0; w < kWords; ++w)
                        for (; unc[w] && before < done + kItems; unc[w] &= unc[w] - 1u)
                            item_s[warp][before++ - done] = (uint16_t)(lane * kTB + w * 32 + __ffs(unc[w]) - 1);
                    __syncwarp();
                    for (int t = lane; t < min(kItems, total - done); t += 32) {
                        const int it = item_s[warp][t], l = it / kTB, j = it % kTB;
                        const float s = dot_seq(R.p + (int64_t)j * R.ld,
                                                a.x.p + (v0 + (warp & 3) * 32 + l) * a.x.ld, R.dim, vec);
                        if (s > 0.0f) atomicOr(&fix_s[warp][l * kWords + (j >> 5)], 1u << (j & 31));
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int w = 0; w < kWords; ++w) word[w] = fix_s[warp][lane * kWords + w];
                __syncwarp();
            }
            if (v < a.x.count) {
                uint32_t* out = a.codes + v * a.ldc + group * kWords;
#pragma unroll
                for (int w = 0; w < kWords; ++w)
                    if (w < nw) out[w] = word[w];
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (a.tensor && warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512) : "memory");
    sum_left(left_s, reinterpret_cast<float*>(smem));  // the ring's memory is free now
}

song_status fail(song_status s, const char* msg) { return song::set_error(s, msg); }

song_status cuda_fail(cudaError_t e, const char* what) {
    char buf[256];
    std::snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
    return song::set_error(SONG_ERR_CUDA, buf);
}

song_status check_shape(int dim, int hash_bits, int64_t n) {
    if (dim < 1) return fail(SONG_ERR_INVALID_ARG, "dim must be >= 1");
    if (hash_bits < 32 || hash_bits % 32 != 0)
        return fail(SONG_ERR_INVALID_ARG, "hash_bits must be a positive multiple of 32");
    if (n < 0) return fail(SONG_ERR_INVALID_ARG, "n must be >= 0");
    return SONG_OK;
}

}  // namespace

namespace song {

cudaError_t launch_bithash(const float* d_R, int dim, int hash_bits, const float* d_x, int64_t n,
                           int64_t ldx, uint32_t* d_codes, int64_t ldc, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    int dev = 0, num_sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    BhArgs a;
    a.R = Rows{d_R, dim, hash_bits, dim, (reinterpret_cast<uintptr_t>(d_R) & 15u) == 0 && dim % 4 == 0};
    a.x = Rows{d_x, ldx, n, dim, (reinterpret_cast<uintptr_t>(d_x) & 15u) == 0 && ldx % 4 == 0};
    a.codes = d_codes;
    a.ldc = ldc;
    a.words = hash_bits / 32;
    a.groups = (a.words + kWords - 1) / kWords;
    a.tensor = dim <= kTensorDim;
    a.tv = kTV;
    if (!a.tensor) {
        // the height with the least time: tiles of the busiest CTA, each as long as
        // its height and about 96 more (the chunks' loads and barriers: 1,000 x
        // 100,000 -> 256 bits 21.4 ms at 128, 12.1 at 32; 10,000 x 6,000 2.5 ms at
        // 128, two tiles, 3.2 at 64, three)
        const int64_t ctas = std::max(1, num_sms / a.groups);
        auto cost = [&](int tv) { return ((n + tv - 1) / tv + ctas - 1) / ctas * (tv + 96); };
        for (int tv = kTV / 2; tv >= 32; tv /= 2)
            if (cost(tv) < cost(a.tv)) a.tv = tv;
    }
    a.tiles = (n + a.tv - 1) / a.tv;
    a.per_group = (int)std::min<int64_t>(std::max(1, num_sms / a.groups), a.tiles);
    a.nch = (dim + kDC - 1) / kDC;
    a.factor = error_factor(dim);
    const bool res = a.nch <= kResChunks;
    const size_t smem = res ? (size_t)(2 * a.nch + 2 * kStagesRes) * kBlock : (size_t)4 * kStagesStream * kBlock;
    void (*kern)(const BhArgs) = res ? bithash_kernel<true> : bithash_kernel<false>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(a.per_group * a.groups), kThreads, smem, st>>>(a);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

}  // namespace song

extern "C" {

song_status song_bithash_matrix(int dim, int hash_bits, unsigned seed, float* R) {
    if (song_status s = check_shape(dim, hash_bits, 0)) return s;
    if (R == nullptr) return fail(SONG_ERR_INVALID_ARG, "R is NULL");
    // The reference's generator and distribution (bitHash.h:23-27), called,
    // not restated: the same standard library gives the same matrix.
    std::mt19937 rng(seed);
    std::normal_distribution<float> gauss(0.0f, 1.0f);
    const size_t total = (size_t)hash_bits * (size_t)dim;
    for (size_t i = 0; i < total; ++i) R[i] = gauss(rng);
    return SONG_OK;
}

song_status song_bithash_project_device(const float* d_R, int dim, int hash_bits,
                                        const float* d_x, int64_t n, int64_t ldx,
                                        uint32_t* d_codes, int64_t ldc, void* stream) {
    if (song_status s = check_shape(dim, hash_bits, n)) return s;
    if (n == 0) return SONG_OK;
    if (d_R == nullptr || d_x == nullptr || d_codes == nullptr)
        return fail(SONG_ERR_INVALID_ARG, "R, x or codes is NULL");
    if (ldx < dim) return fail(SONG_ERR_INVALID_ARG, "ldx must be >= dim");
    if (ldc < hash_bits / 32) return fail(SONG_ERR_INVALID_ARG, "ldc must be >= hash_bits / 32");
    if ((n + 63) / 64 > (int64_t)INT32_MAX)
        return fail(SONG_ERR_INVALID_ARG, "n too large for one launch");
    cudaError_t e = song::launch_bithash(d_R, dim, hash_bits, d_x, n, ldx, d_codes, ldc,
                                         (cudaStream_t)stream);
    if (e != cudaSuccess) return cuda_fail(e, "bithash launch");
    return SONG_OK;
}

song_status song_bithash_project(const float* R, int dim, int hash_bits, const float* x,
                                 int64_t n, uint32_t* codes) {
    if (song_status s = check_shape(dim, hash_bits, n)) return s;
    if (n == 0) return SONG_OK;
    if (R == nullptr || x == nullptr || codes == nullptr)
        return fail(SONG_ERR_INVALID_ARG, "R, x or codes is NULL");
    const int words = hash_bits / 32;
    float* d_R = nullptr;
    float* d_x = nullptr;
    uint32_t* d_c = nullptr;
    cudaStream_t st = nullptr;
    const size_t rb = (size_t)hash_bits * dim * 4, xb = (size_t)n * dim * 4,
                 cb = (size_t)n * words * 4;
    cudaError_t e = song::device_alloc((void**)&d_R, rb);
    if (e == cudaSuccess) e = song::device_alloc((void**)&d_x, xb);
    if (e == cudaSuccess) e = song::device_alloc((void**)&d_c, cb);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_R, R, rb, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_x, x, xb, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = song::launch_bithash(d_R, dim, hash_bits, d_x, n, dim, d_c, words, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(codes, d_c, cb, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_R);
    cudaFree(d_x);
    cudaFree(d_c);
    if (st) cudaStreamDestroy(st);
    if (e == cudaErrorMemoryAllocation) return fail(SONG_ERR_OOM, "bithash: device allocation failed");
    if (e != cudaSuccess) return cuda_fail(e, "bithash");
    return SONG_OK;
}

}  // extern "C"

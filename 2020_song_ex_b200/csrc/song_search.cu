// song_search.cu -- row conversions and search launches (the kernels are in
// song_search.cuh, their instances in song_search_*.cu).
#include "song_search.cuh"

#include <cstring>

namespace song {

std::atomic<int64_t> g_launches{0};

namespace {

// FP32 rows of integers in [0, 255] -> byte rows, zero padded to out_ld bytes.
__global__ void rows_to_u8(const float* __restrict__ x, int64_t n, int dim, int ld,
                           uint8_t* __restrict__ out, int out_ld) {
    const int64_t r = blockIdx.x;
    if (r >= n) return;
    for (int i = threadIdx.x; i < out_ld; i += blockDim.x)
        out[r * out_ld + i] = i < dim ? (uint8_t)x[r * ld + i] : (uint8_t)0;
}

// Order-preserving map of a float to an int, for atomicMin / atomicMax.
__device__ __forceinline__ int ord_int(float x) {
    const int b = __float_as_int(x);
    return b >= 0 ? b : b ^ 0x7fffffff;
}

// out[0] := 1 if some value is not an integer of magnitude below 2^24, out[1]
// and out[2] the smallest and largest value in ord_int order (of the values
// before the first block saw such a one).  One pass over the rows.
__global__ void scan_rows(const float* __restrict__ x, int64_t n, int dim, int ld, int* __restrict__ out) {
    float lo = INFINITY, hi = -INFINITY;
    bool bad = false;
    const int64_t total = n * (int64_t)dim, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
        const float v = __ldg(x + (ld == dim ? i : (i / dim) * ld + i % dim));
        bad |= !(v == rintf(v)) || !(fabsf(v) < 16777216.0f);
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
    }
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(FULL, lo, w));
        hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, w));
    }
    bad = __any_sync(FULL, bad);
    if ((threadIdx.x & 31) == 0) {
        if (bad) {
            out[0] = 1;
        } else {
            atomicMin(out + 1, ord_int(lo));
            atomicMax(out + 2, ord_int(hi));
        }
    }
}

// FP32 -> BF16 (round to nearest even) rows, zero padded to out_ld bytes.
__global__ void quantize_bf16(const float* __restrict__ x, int64_t n, int dim, int ld,
                              unsigned short* __restrict__ out, int out_ld) {
    const int64_t r = blockIdx.x;
    if (r >= n) return;
    const int pd = out_ld / 2;
    for (int i = threadIdx.x; i < pd; i += blockDim.x) {
        const float v = i < dim ? x[r * ld + i] : 0.0f;
        out[r * pd + i] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
    }
}

// FP32 -> FP8 e4m3 rows with scale amax/448 (448 = largest finite e4m3):
// x ~= scale * e4m3(x / scale); one warp per row.
__global__ void quantize_fp8(const float* __restrict__ x, int64_t n, int dim, int ld,
                             unsigned char* __restrict__ out, int out_ld,
                             float* __restrict__ scales) {
    const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    float amax = 0.0f;
    for (int i = lane; i < dim; i += 32) amax = fmaxf(amax, fabsf(x[r * ld + i]));
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) amax = fmaxf(amax, __shfl_xor_sync(FULL, amax, w));
    const float scale = amax > 0.0f ? amax / 448.0f : 1.0f;
    const float inv = 1.0f / scale;
    for (int i = lane; i < out_ld; i += 32) {
        const float v = i < dim ? x[r * ld + i] * inv : 0.0f;
        out[r * out_ld + i] = (unsigned char)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
    }
    if (lane == 0) scales[r] = scale;
}

KernelSel pick_kernel(int kind, const SearchArgs& a, bool reg) {
    if (a.lm != 0) return kind == SONG_KIND_L2 ? pick_learned(a, reg) : KernelSel();
    if (kind != SONG_KIND_L2) return pick_hamming(a, reg);
    return a.prec != SONG_PREC_FP32 ? pick_lowp(a, reg) : pick_l2(a, reg);
}

// Resident CTAs per SM of a TMEM-id kernel.  The runtime's occupancy query
// reports a single CTA per SM for kernels that allocate tensor memory, yet
// several such CTAs run side by side when their registers, shared memory and
// TMEM columns fit, so the limit is computed from those resources: registers
// are allocated per warp in units of 8 per thread out of 16,384 per SM
// sub-partition (four per SM), shared memory per CTA includes the runtime's
// reservation, and each SM has 512 TMEM columns.  A CTA beyond what fits
// would only wait in tcgen05.alloc for an earlier one to finish.
cudaError_t tm_ctas_per_sm(KernelFn fn, int dev, int warps, size_t dyn_smem, int tm_cols, int* out) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return e;
    int smem_sm = 0, reserved = 0, regs_sm = 0, max_blocks = 0, max_threads = 0;
    e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&max_blocks, cudaDevAttrMaxBlocksPerMultiprocessor, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&max_threads, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
    if (e != cudaSuccess) return e;
    const size_t cta_smem = dyn_smem + fa.sharedSizeBytes + (size_t)reserved;
    const int by_smem = (int)((size_t)smem_sm / cta_smem);
    const int warp_regs = ((fa.numRegs + 7) / 8) * 8 * 32;
    const int warps_per_quarter = warp_regs > 0 ? (regs_sm / 4) / warp_regs : 64;
    const int by_regs = (warps_per_quarter * 4) / warps;
    const int by_threads = max_threads / (warps * 32);
    const int by_tmem = 512 / tm_cols;
    *out = std::min(std::min(std::min(by_smem, by_regs), std::min(by_threads, max_blocks)), by_tmem);
    return cudaSuccess;
}

// Per-warp shared memory of the TMEM-id kernels: [query if kept in shared
// memory][32-entry row list][candidate distances][candidate ids, unless they
// are in TMEM too][result distances][Bloom filter], the Bloom region being at
// least cap ints because finish() may keep the extracted slots there once
// the search is over.
void tm_layout(int query_floats, bool cand_in_tmem, bool res_d_in_tmem, SearchArgs* a) {
    const int capr = round_up(a->cap, 32);
    a->q_off = 0;
    a->rows_off = round_up(query_floats * 4, 16);
    // the row list doubles as the push stage: 32 ids, and 32 distances when
    // the result distances are in TMEM
    a->cd_off = a->rows_off + (res_d_in_tmem ? 256 : 128);
    int off = a->cd_off + capr * 4;
    a->ci_off = 0;
    if (!cand_in_tmem) {
        a->ci_off = off;
        off += capr * 4;
    }
    a->rd_off = 0;
    if (!res_d_in_tmem) {
        a->rd_off = off;
        off += capr * 4;
    }
    a->ri_off = 0;
    a->bl_off = round_up(off, 16);
    a->warp_smem = round_up(a->bl_off + std::max(a->bf_words * 8, capr * 4), 16);
    a->tm_warp_cols = ((cand_in_tmem ? 1 : 0) + 1 + (res_d_in_tmem ? 1 : 0)) * (capr / 32);
}

// Per-warp shared memory of the register-queue kernels: [query if kept in
// shared memory][32-entry row list][candidate ids][result ids][Bloom filter],
// the Bloom region being at least 2 cap ints, the scratch of finish().
void reg_layout(int query_floats, SearchArgs* a) {
    const int capr = round_up(a->cap, 32);
    a->q_off = 0;
    a->rows_off = round_up(query_floats * 4, 16);
    a->ci_off = a->rows_off + 128;
    a->ri_off = a->ci_off + capr * 4;
    a->bl_off = a->ri_off + capr * 4;
    a->cd_off = a->rd_off = 0;
    a->warp_smem = round_up(a->bl_off + std::max(a->bf_words * 8, 2 * capr * 4), 16);
}

}  // namespace

int u8_row_bytes(int dim) { return round_up(dim, 16); }

cudaError_t convert_rows_u8(const float* d_rows, int64_t n, int dim, int ld, uint8_t* d_out,
                            int out_ld, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    rows_to_u8<<<(unsigned)n, 128, 0, st>>>(d_rows, n, dim, ld, d_out, out_ld);
    return cudaGetLastError();
}

cudaError_t scan_base_range(const float* d_rows, int64_t n, int dim, int ld, int* d_scratch,
                            cudaStream_t st, BaseRange* r) {
    *r = BaseRange();
    if (n <= 0 || dim <= 0) return cudaSuccess;
    int h[3] = {0, INT_MAX, INT_MIN};
    cudaError_t e = cudaMemcpyAsync(d_scratch, h, sizeof h, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const int64_t blocks = std::min<int64_t>((n * (int64_t)dim + 255) / 256, 148 * 8);
    scan_rows<<<(unsigned)blocks, 256, 0, st>>>(d_rows, n, dim, ld, d_scratch);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_scratch, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess || h[0] != 0) return e;
    auto value = [](int o) {
        const int b = o >= 0 ? o : o ^ 0x7fffffff;
        float f;
        std::memcpy(&f, &b, sizeof f);
        return f;
    };
    r->int_base = 1;
    r->lo = value(h[1]);
    r->hi = value(h[2]);
    return cudaSuccess;
}

int search_row_stride(int kind, int dim) {
    if (kind == SONG_KIND_L2) return round_up(dim, 4);
    if (dim <= 4) return 4;
    if (dim <= 8) return 8;
    if (dim <= 16) return 16;
    return 32;
}

int lowp_padded_dim(int prec, int dim) {
    const int unit = prec == SONG_PREC_BF16 ? 64 : 128;  // 8 lanes x 16 B per pass over a row
    return round_up(dim, unit);
}

cudaError_t quantize_rows(int prec, const float* d_rows, int64_t n, int dim, int ld, void* d_out,
                          int out_ld, float* d_scales, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (prec == SONG_PREC_BF16) {
        quantize_bf16<<<(unsigned)n, 128, 0, st>>>(d_rows, n, dim, ld,
                                                   static_cast<unsigned short*>(d_out), out_ld);
    } else if (prec == SONG_PREC_FP8) {
        quantize_fp8<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(
            d_rows, n, dim, ld, static_cast<unsigned char*>(d_out), out_ld, d_scales);
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

int search_warp_smem(int kind, int dim, int cap, int bf_words, SearchArgs* a) {
    (void)kind;
    const int capr = round_up(cap, 32);
    a->q_off = 0;
    a->rows_off = round_up(dim * 4, 16);
    a->cd_off = a->rows_off + 128;
    a->ci_off = a->cd_off + capr * 4;
    a->rd_off = a->ci_off + capr * 4;
    a->ri_off = a->rd_off + capr * 4;
    a->bl_off = round_up(a->ri_off + capr * 4, 16);
    a->warp_smem = round_up(a->bl_off + bf_words * 8, 16);
    return a->warp_smem;
}

static cudaError_t launch_instance(KernelSel ks, int kind, const SearchArgs& args, int num_sms,
                                   cudaStream_t stream) {
    if (ks.fn == nullptr) return cudaErrorInvalidValue;
    if (args.trace == nullptr && ks.fn_nt != nullptr) {
        ks.fn = ks.fn_nt;
        ks.fn_tmc = ks.fn_tmc_nt;
        ks.fn_tmd = ks.fn_tmd_nt;
    }
    KernelFn fn = ks.fn;
    SearchArgs a = args;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int smem_optin = 0;
    e = cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    int warps;
    int tm_per_sm = 0;
    if (ks.qr) {
        warps = ks.threads / 32;
        reg_layout(ks.query_smem ? a.qdim : 0, &a);
    } else if (ks.tm) {
        // ids in TMEM: CTAs of 4 warps, one per lane quarter; ceil(cap/32)
        // columns per warp and queue, allocated per CTA in a power of two >= 32.
        // The candidate ids go to shared memory unless that costs resident CTAs
        // (large queues and Bloom filters), then to TMEM as well.
        warps = ks.threads / 32;
        auto shape = [&](KernelFn f, bool cand_tm, bool res_d_tm, SearchArgs* s2, int* per_sm) -> cudaError_t {
            tm_layout(ks.query_smem ? s2->qdim : 0, cand_tm, res_d_tm, s2);
            int cols = 32;
            while (cols < s2->tm_warp_cols * (warps / 4)) cols <<= 1;
            s2->tm_cols = cols;
            *per_sm = 0;
            if (cols > 512 || (size_t)warps * s2->warp_smem > (size_t)smem_optin) return cudaSuccess;
            return tm_ctas_per_sm(f, dev, warps, (size_t)warps * s2->warp_smem, cols, per_sm);
        };
        // the layout with the most resident CTAs; on a tie the one with fewer
        // TMEM accesses (ids, then distances, in shared memory)
        SearchArgs a0 = a, a1 = a, a2 = a;
        int p0 = 0, p1 = 0, p2 = 0;
        e = shape(ks.fn, false, false, &a0, &p0);
        if (e == cudaSuccess) e = shape(ks.fn_tmc, true, false, &a1, &p1);
        if (e == cudaSuccess && ks.fn_tmd != nullptr) e = shape(ks.fn_tmd, true, true, &a2, &p2);
        if (e != cudaSuccess) return e;
        a = a0;
        tm_per_sm = p0;
        // (all of them, when the launch fits without more residency: 5 % at 1,000
        // queries and ef 576)
        const bool all_resident = ((int64_t)args.nq + warps - 1) / warps <= (int64_t)p0 * num_sms;
        if (!all_resident && p1 > tm_per_sm) {
            a = a1;
            fn = ks.fn_tmc;
            tm_per_sm = p1;
        }
        if (!all_resident && p2 > tm_per_sm) {
            a = a2;
            fn = ks.fn_tmd;
            tm_per_sm = p2;
        }
        // four such warps leave no room for the query: the instances that read it
        // from global memory
        if (tm_per_sm < 1 && ks.query_smem && kind == SONG_KIND_L2 && a.prec == SONG_PREC_FP32 &&
            args.dim <= kU8MaxDim)
            return launch_instance(pick_l2(args, false, true), kind, args, num_sms, stream);
        if (tm_per_sm < 1) return cudaErrorInvalidConfiguration;
    } else {
        // Up to 8 warps per CTA while the CTA's shared memory stays within a
        // quarter of the opt-in limit, so several CTAs can share an SM.
        warps = ks.threads / 32;
        while (warps > 1 && (size_t)warps * a.warp_smem > (size_t)smem_optin / 4) warps >>= 1;
    }
    const size_t smem = (size_t)warps * a.warp_smem;
    if (smem > (size_t)smem_optin) return cudaErrorInvalidConfiguration;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if (ks.tm) {
        per_sm = tm_per_sm;
    } else {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, warps * 32, smem);
    }
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int64_t need = ((int64_t)a.nq + warps - 1) / warps;
    const int grid = (int)std::min<int64_t>((int64_t)per_sm * num_sms, need);
    // Plain searches (no learned stage, no caller seeds: nothing they read
    // can come from the launch before them) with a self-resetting counter
    // may overlap the previous search launch's tail on the same stream.
    const bool overlap = a.done != nullptr && a.lm == 0 && a.qseeds == nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)(warps * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, fn, a);
    if (e != cudaSuccess) return e;
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

constexpr int kRegAlways = 5;  // registers per lane and queue

cudaError_t launch_search(int kind, const SearchArgs& args, int num_sms, cudaStream_t stream) {
    if (args.nq <= 0) return cudaSuccess;
    // Queues in registers, unless they are too long or four warps' filters and
    // ids do not fit in shared memory.  Up to 160 slots they are faster at any
    // number of queries (10,000 of 128 integers: ef 64 1.29 -> 1.09 ms, ef 128
    // 2.07 -> 1.95, ef 150 2.30 -> 2.25; one at ef 150 611 -> 511 us; 60, 120 and
    // 150 slots and 1 to 10,000 queries of the other row types, too: float 1-33 %,
    // BF16 and FP8 up to 10 %, Hamming 7-23 %, learned 5-36 %).  Up to 256 the work per
    // operation passes that of the group summaries and only the shorter chain
    // remains, which wins while the SMs are nearly empty.  200 and 256 slots, 1 to
    // 592 queries / 10,000, time of the others over theirs: 128 integers 1.04-1.07
    // / 0.87, float rows 1.12-1.22 / 0.99-1.01, BF16 1.02 / 0.98, FP8 1.00 / 0.97,
    // Hamming 1.08-1.12 / 0.90-0.92, learned integers 1.05-1.08 / 0.94, learned
    // float rows 0.98-1.00 / 1.01, learned BF16 1.04-1.05 / 1.08.
    const KernelSel reg = pick_kernel(kind, args, true);
    if (reg.fn != nullptr) {
        SearchArgs a = args;
        reg_layout(reg.query_smem ? a.qdim : 0, &a);
        int dev = 0, optin = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e != cudaSuccess) return e;
        const int warps = reg.threads / 32;
        const bool fits = (size_t)warps * a.warp_smem <= (size_t)optin;
        const bool few = ((int64_t)args.nq + warps - 1) / warps <= num_sms;
        if (fits && (reg.qr <= kRegAlways || few)) return launch_instance(reg, kind, args, num_sms, stream);
    }
    return launch_instance(pick_kernel(kind, args, false), kind, args, num_sms, stream);
}

}  // namespace song

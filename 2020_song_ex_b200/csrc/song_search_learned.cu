// song_search_learned.cu -- instances of the learned search, the trace pass of
// its training, and the serving kernel.
#include "song_search.cuh"

namespace song {

namespace {

#include "song_serve_kernel.inc"

// Training traces (lm 1) keep the queues in shared memory.
template <int NE, int DT, int LM>
KernelSel sel(const SearchArgs& a, bool reg) {
    if constexpr (LM != 1) {
        if (reg) return reg_queues<0, NE, DT, LM>(a);
    }
    return reg ? KernelSel() : ksel<0, NE, 1, DT, LM>();
}

template <int LM>
KernelSel by_rows(const SearchArgs& a, bool reg) {
    if (a.prec == SONG_PREC_BF16) return sel<0, SONG_PREC_BF16, LM>(a, reg);
    if (a.prec == SONG_PREC_FP8) return sel<0, SONG_PREC_FP8, LM>(a, reg);
    if (a.u8 != nullptr && a.dim <= 128) return sel<-1, 0, LM>(a, reg);
    return sel<0, 0, LM>(a, reg);
}

}  // namespace

KernelSel pick_learned(const SearchArgs& a, bool reg) {  // L2, queues up to 1024 slots
    if (a.cap > 1024) return KernelSel();
    if (a.lm == 1) return by_rows<1>(a, reg);
    // a stop model that can never fire (none, or threshold >= 1): the entry-only
    // instance, without the stop statistics -- the same results, less state
    if (a.stop_w == nullptr || !(a.stop_thr < INFINITY)) return by_rows<3>(a, reg);
    return by_rows<2>(a, reg);
}

cudaError_t launch_serve(const ServeArgs& s, int num_sms, int max_ctas, int reserve_sms,
                         cudaStream_t st, int* warps_out) {
    using ServeFn = void (*)(const ServeArgs);
    ServeFn fn;
    const SearchArgs& a = s.base;
    if (a.prec == SONG_PREC_BF16) fn = serve_kernel<0, SONG_PREC_BF16>;
    else if (a.prec == SONG_PREC_FP8) fn = serve_kernel<0, SONG_PREC_FP8>;
    else if (a.u8 != nullptr && a.dim <= 128) fn = serve_kernel<-1, 0>;
    else fn = serve_kernel<0, 0>;
    int dev = 0, optin = 0, smem_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (e != cudaSuccess) return e;
    int warps;
    size_t smem;
    if (reserve_sms > 0 && reserve_sms < num_sms) {
        // Leave reserve_sms SMs free for the batched entry stage: one CTA of up
        // to 16 warps per SM, its shared memory padded past half of the SM so
        // that no SM can hold two, on num_sms - reserve_sms SMs.
        warps = 16;
        while (warps > 1 && (size_t)warps * a.warp_smem > (size_t)optin) warps >>= 1;
        smem = std::max<size_t>((size_t)warps * a.warp_smem, (size_t)smem_sm / 2 + 1024);
        if (smem > (size_t)optin) return cudaErrorInvalidConfiguration;
    } else {
        warps = 8;
        while (warps > 1 && (size_t)warps * a.warp_smem > (size_t)optin / 4) warps >>= 1;
        smem = (size_t)warps * a.warp_smem;
        if (smem > (size_t)optin) return cudaErrorInvalidConfiguration;
    }
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, warps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    int grid = per_sm * num_sms;
    if (reserve_sms > 0 && reserve_sms < num_sms) grid = num_sms - reserve_sms;  // per_sm is 1
    if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
    fn<<<grid, warps * 32, smem, st>>>(s);
    if (warps_out) *warps_out = grid * warps;
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

}  // namespace song

// song_search_l2.cu -- plain FP32 search instances.
#include "song_search.cuh"

namespace song {

namespace {
template <int KIND, int NE, int DT>
KernelSel by_cap(const SearchArgs& a, bool reg) {
    if (reg) return reg_queues<KIND, NE, DT, 0>(a);
    if (a.cap <= 1024) return ksel<KIND, NE, 1, DT>();
    if (a.cap <= 2048) return ksel<KIND, NE, 2, DT>();
    if (a.cap <= 4096) return ksel<KIND, NE, 4, DT>();
    return KernelSel();
}
}  // namespace

KernelSel pick_l2(const SearchArgs& a, bool reg) {
    // an index with byte rows: the byte-row instances
    if (a.u8 != nullptr && a.dim <= 128) return by_cap<0, -1, 0>(a, reg);
    if (a.u8 != nullptr && a.dim <= 256) return by_cap<0, -2, 0>(a, reg);
    return by_cap<0, 0, 0>(a, reg);
}

}  // namespace song

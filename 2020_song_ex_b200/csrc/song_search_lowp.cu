// song_search_lowp.cu -- instances of the precision form.
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

KernelSel pick_lowp(const SearchArgs& a, bool reg) {
    if (a.prec == SONG_PREC_BF16) return by_cap<0, 0, SONG_PREC_BF16>(a, reg);
    if (a.prec == SONG_PREC_FP8) return by_cap<0, 0, SONG_PREC_FP8>(a, reg);
    return KernelSel();
}

}  // namespace song

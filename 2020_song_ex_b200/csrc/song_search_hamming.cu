// song_search_hamming.cu -- Hamming search instances.
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

KernelSel pick_hamming(const SearchArgs& a, bool reg) {
    switch (a.ld) {
        case 4: return by_cap<1, 1, 0>(a, reg);
        case 8: return by_cap<1, 2, 0>(a, reg);
        case 16: return by_cap<1, 4, 0>(a, reg);
        case 32: return by_cap<1, 8, 0>(a, reg);
        default: return KernelSel();
    }
}

}  // namespace song

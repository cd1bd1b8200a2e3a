// song_search_hamming.cu -- Hamming search instances.
#include "song_search.cuh"

namespace song {

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

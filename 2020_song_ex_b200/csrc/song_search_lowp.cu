// song_search_lowp.cu -- instances of the precision form.
#include "song_search.cuh"

namespace song {

KernelSel pick_lowp(const SearchArgs& a, bool reg) {
    if (a.prec == SONG_PREC_BF16) return by_cap<0, 0, SONG_PREC_BF16>(a, reg);
    if (a.prec == SONG_PREC_FP8) return by_cap<0, 0, SONG_PREC_FP8>(a, reg);
    return KernelSel();
}

}  // namespace song

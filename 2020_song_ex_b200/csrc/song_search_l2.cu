// song_search_l2.cu -- plain FP32 search instances.
#include "song_search.cuh"

namespace song {

KernelSel pick_l2(const SearchArgs& a, bool reg, bool query_global) {
    // an index with byte rows: the byte-row instances, which read a query that is
    // not whole numbers from global memory (any query of an index without them)
    const bool bytes = a.u8 != nullptr || query_global;
    if (bytes && a.dim <= 128) return by_cap<0, -1, 0>(a, reg);
    if (bytes && a.dim <= 256) return by_cap<0, -2, 0>(a, reg);
    return by_cap<0, 0, 0>(a, reg);
}

}  // namespace song

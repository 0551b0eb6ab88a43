// limits.h -- host checks of counts against 32-bit indices (no CUDA).
#pragma once
#include <cstdint>

namespace tsr {

// Entries of the neighbour rows of a graph of `edges` edges: an edge has one in
// the row of either end.  False where the rows' 32-bit offsets cannot address
// them (a sum of the row lengths in 32 bits would have wrapped); the six edge
// events of a leaf alone, below 2^32, do not rule that out.
inline bool neighbor_entries(uint64_t edges, uint32_t *entries) {
    if (2 * edges >= 0xFFFFFFFFull) return false;
    *entries = (uint32_t)(2 * edges);
    return true;
}

}  // namespace tsr

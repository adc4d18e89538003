// cast_queue.h - the 32-ray chunks a warp of cast_persistent_kernel walks, for any 32-bit
// number of rays n (the sums stay below 2^32).
#pragma once

#include "vrt_internal.h"

namespace vrt {

// The end of the chunk that starts at ray `first` < n.
VRT_HD inline uint32_t chunk_end(uint32_t first, uint32_t n) {
    return n - first < 32u ? n : first + 32u;
}
// The warp's next chunk, `stride` rays on; n or more when there is none.
VRT_HD inline uint32_t chunk_after(uint32_t first, uint32_t stride, uint32_t n) {
    return n - first <= stride ? n : first + stride;
}

}  // namespace vrt

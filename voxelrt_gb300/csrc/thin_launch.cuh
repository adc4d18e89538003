// Frames, small ones with fewer rays per warp (launch_rules.h).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "launch_rules.h"

namespace vrt {

// The pixel of this thread in such a launch's frame: blocks of kFrameThreads, two by two warps, each
// an area of 2^lanes_log2 pixels (8x4 for 32).  One above the other, two warps a block: 118.3 us for a
// 1080p frame with sun rays against 117.4, 35.1 against 34.7 for a 720p G-buffer, and 198
// against 188 for 1024x1024 anisotropic paths, whose blocks fill an 8 KB table each.  False for a
// lane without a pixel.  kThin: fewer than 32, an instantiation of its own where the test costs
// the large launches (1 % of a 720p G-buffer).
constexpr uint32_t kFrameThreads = 128;
template <bool kThin>
__device__ __forceinline__ bool thin_pixel(uint32_t lanes_log2, uint32_t& px, uint32_t& py) {
    if (!kThin) lanes_log2 = 5;
    const uint32_t lane = threadIdx.x & 31, wl = (lanes_log2 + 1) / 2;
    px = ((blockIdx.x * 2 + ((threadIdx.x >> 5) & 1u)) << wl) + (lane & ((1u << wl) - 1u));
    py = ((blockIdx.y * 2 + (threadIdx.x >> 6)) << (lanes_log2 - wl)) + (lane >> wl);
    return (lane >> lanes_log2) == 0;
}
inline dim3 thin_grid(uint32_t lanes_log2, uint32_t width, uint32_t height) {
    const uint32_t wl = (lanes_log2 + 1) / 2, tw = 2u << wl, th = 2u << (lanes_log2 - wl);
    return dim3((width + tw - 1) / tw, (height + th - 1) / th);
}

}  // namespace vrt

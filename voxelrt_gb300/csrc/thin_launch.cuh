// Small launches: fewer rays per warp.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace vrt {

// Rays per warp of a small launch (log2, 2..5): as few as keep the launch within kThinWarps warps.
// A launch that leaves most of the chip idle lasts as long as its longest ray, and a ray's
// step waits for the slowest lane of its warp: with 4 rays a warp a 64x64 frame of a
// 256-voxel terrain takes 12.5 us against 14.5, 2,000 random rays 16.4 us against 18.6 (two rays a
// warp: another 2 % at 1,000 to 2,000 rays, nothing elsewhere).  64x64 paths of the terrain: sun
// rays 20.1 -> 17.4 us, 3 bounces 41.4 -> 28.9, anisotropic with both 51.4 -> 34.3; G-buffers
// 15.3 -> 12.5.  kThinWarps where the gain ends (with 1,216 frames of 100x100 to 160x160 take 2 to 7 %
// more, such paths 5 to 12 %; with 4,864 paths whose rays end at once up to half as much again).
constexpr uint32_t kThinWarps = 2432;
inline uint32_t thin_lanes_log2(uint64_t rays) {
    uint32_t l = 5;
    while (l > 2 && rays >> (l - 1) <= kThinWarps) l--;
    return l;
}

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

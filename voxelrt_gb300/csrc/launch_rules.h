// launch_rules.h - how small launches are spread over the chip: rays per warp and claims per tile,
// by the number of SMs (152 on GB300: 2,432 warps, 7,296 tiles).
#pragma once

#include <cstdint>

namespace vrt {

// SMs of the calling thread's current device (world.cu).
uint32_t sm_count();

// Rays per warp of a small launch (log2, 2..5): as few as keep the launch within kThinWarps warps a SM.
// A launch that leaves most of the chip idle lasts as long as its longest ray, and a ray's
// step waits for the slowest lane of its warp.  Kernel times in a graph of 40 launches (event times of
// single launches end in the launch itself, 3 to 4 us, and in steps of 1 to 2 us): 64x64 paths of a
// 256-voxel terrain with 4 rays a warp 10.1 us against 12.6, with sun rays 17.3 against 22.6, with 2
// bounces 28.7 against 44.2, anisotropic 10.6 / 19.5 / 25.9 against 13.7 / 23.6 / 40.2; 2,000 random rays
// 16.4 us against 18.6 (two rays a warp: another 2 % at 1,000 to 2,000 rays, nothing elsewhere).
// kThinWarps where the gain ends: with 8 a SM paths of 100x90 to 200x190 take up to 25 % more, with 32
// paths whose rays end at once up to half as much again.  From within a solid voxel, where every ray
// ends on its first step, it costs 0.1 to 0.4 us of 2 to 4 (100x90: 2.1 -> 2.4 us, sun rays 2.6 ->
// 3.1).
constexpr uint32_t kThinWarps = 16;
inline uint32_t thin_lanes_log2(uint64_t rays, uint32_t sms) {
    uint32_t l = 5;
    while (l > 2 && rays >> (l - 1) <= (uint64_t)kThinWarps * sms) l--;
    return l;
}

// Claims per tile (log2) of a batch whose chunks are one tile of 64 rays: a launch of few tiles leaves
// most of the chip idle, and a warp that traces 64 rays takes twice as long as one with 32.
// Half tiles up to kHalfTiles tiles a SM (two 640x360 views of a terrain, 7,200 tiles, 39.3 us against 45.8
// whole; from within a dense world 20.6 against 17.0).  Launches with bounces take half tiles at any
// size, as their warps end far apart (two 720p views of 4 bounces 372 -> 355 us, 1024x1024 131 -> 118;
// quarter tiles 370 and 133 us).  Below kThinWarps warps a SM also fewer rays a warp, down to 4, as
// above (64x64 terrain views: primary rays 25.1 -> 17.7 us, 3 bounces 68 -> 36, anisotropic with sun
// rays and bounces 86 -> 40; with twice as many warps faster still there by 2 to 4 us, and slower by
// as much where rays end at once).
constexpr uint32_t kHalfTiles = 48;
inline uint32_t claim_split_log2(uint32_t tiles, bool bounces, uint32_t sms) {
    // (the queue counts claims in 32 bits)
    if (tiles > (bounces ? 1u << 30 : kHalfTiles * sms)) return 0;
    uint32_t s = 1;
    while (s < 4 && (uint64_t)tiles << (s + 1) <= (uint64_t)kThinWarps * sms) s++;
    return s;
}

}  // namespace vrt

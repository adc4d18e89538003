// edit_geometry.h - which bricks an edit's sphere reaches (host).
#pragma once

#include <algorithm>
#include <cstdint>

#include "vrt_internal.h"

namespace vrt {

// Closest voxel of the brick to the center lies within the sphere.
inline bool sphere_reaches_brick(const vrt_edit& e, int32_t bx, int32_t by, int32_t bz) {
    const int32_t b[3] = {bx, by, bz};
    int64_t d2 = 0;
    for (int c = 0; c < 3; c++) {
        const int64_t lo = (int64_t)b[c] * 8, hi = lo + 7;
        const int64_t p = std::min(std::max<int64_t>(e.center[c], lo), hi);
        d2 += (p - e.center[c]) * (p - e.center[c]);
    }
    return d2 <= (int64_t)e.radius * e.radius;
}

// The sphere reaches every brick of [lo, hi] in sector `sc`: the farthest of them on each axis.
// (A sphere of radius 400 over a whole world spent 400 us of the host's 470 on its 131,072 bricks.)
inline bool sphere_reaches_all(const vrt_edit& e, const int32_t sc[3], const int32_t lo[3], const int32_t hi[3]) {
    int64_t d2 = 0;
    for (int c = 0; c < 3; c++) {
        const int64_t first = (int64_t)(sc[c] * 4 + lo[c]) * 8, last = (int64_t)(sc[c] * 4 + hi[c]) * 8;
        // to the last voxel of the first brick, to the first voxel of the last one
        const int64_t d = std::max({e.center[c] - (first + 7), last - e.center[c], (int64_t)0});
        d2 += d * d;
    }
    return d2 <= (int64_t)e.radius * e.radius;
}

// Bits of the bricks of a sector whose in-sector coordinates lie in [lo, hi] per axis
// (brick bit x | z<<2 | y<<4).
inline uint64_t box_bits(const int32_t lo[3], const int32_t hi[3]) {
    uint64_t m = 0;
    for (int32_t y = lo[1]; y <= hi[1]; y++)
        for (int32_t z = lo[2]; z <= hi[2]; z++)
            for (int32_t x = lo[0]; x <= hi[0]; x++) m |= 1ull << (x | z << 2 | y << 4);
    return m;
}

}  // namespace vrt

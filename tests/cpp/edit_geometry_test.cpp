// edit_geometry_test.cpp - sphere_reaches_all (edit_geometry.h) against the test of each brick, on
// the host.  Prints FAIL lines and exits non-zero on a mismatch.
#include <cstdio>
#include <random>

#include "edit_geometry.h"

using namespace vrt;

int main() {
    std::mt19937 rng(3);
    int fails = 0, all = 0, some = 0;
    for (int i = 0; i < 400000; i++) {
        vrt_edit e{};
        e.radius = std::uniform_int_distribution<uint32_t>(0, i % 3 ? 60 : 4096)(rng);
        int32_t sc[3], lo[3], hi[3];
        for (int c = 0; c < 3; c++) {
            sc[c] = std::uniform_int_distribution<int32_t>(0, 63)(rng);
            lo[c] = std::uniform_int_distribution<int32_t>(0, 3)(rng);
            hi[c] = std::uniform_int_distribution<int32_t>(lo[c], 3)(rng);
            // a center about as far from the sector as the radius, on every side of it
            const int32_t r = (int32_t)e.radius + 34;
            e.center[c] = sc[c] * 32 + 16 + std::uniform_int_distribution<int32_t>(-r, r)(rng) * (i % 4) / 4;
        }
        bool want = true;
        for (int32_t y = lo[1]; y <= hi[1]; y++)
            for (int32_t z = lo[2]; z <= hi[2]; z++)
                for (int32_t x = lo[0]; x <= hi[0]; x++)
                    want &= sphere_reaches_brick(e, sc[0] * 4 + x, sc[1] * 4 + y, sc[2] * 4 + z);
        (want ? all : some)++;
        if (sphere_reaches_all(e, sc, lo, hi) != want && fails++ < 5)
            std::printf("FAIL center %d %d %d radius %u sector %d %d %d\n", e.center[0], e.center[1], e.center[2], e.radius,
                        sc[0], sc[1], sc[2]);
    }
    if (all < 1000 || some < 1000) fails++;  // both outcomes are met
    std::printf("%s: %d failures\n", fails ? "FAIL" : "ok", fails);
    return fails ? 1 : 0;
}

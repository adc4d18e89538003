// cast_queue_test.cpp - the chunks of cast_persistent_kernel (cast_queue.h) on the host: over
// all warps every ray lies in exactly one chunk, up to the largest 32-bit number of rays.
// Prints FAIL lines and exits non-zero on a mismatch.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <utility>
#include <vector>

#include "cast_queue.h"

using namespace vrt;

// The chunks of `warps` warps over n rays that start at ray `from` or later (from: a multiple of
// a whole stride, so that the test need not walk four thousand million rays).
static int check(uint32_t n, uint32_t warps, uint32_t from) {
    const uint32_t stride = warps * 32;
    std::vector<std::pair<uint32_t, uint32_t>> chunks;
    for (uint32_t g = 0; g < warps; g++) {
        uint32_t next = from / stride * stride;
        if (n - next <= g * 32) continue;
        next += g * 32;
        for (int k = 0; next < n; k++) {
            if (k > 1000) {
                std::printf("FAIL n=%u warps=%u: warp %u does not end\n", n, warps, g);
                return 1;
            }
            chunks.emplace_back(next, chunk_end(next, n));
            next = chunk_after(next, stride, n);
        }
    }
    std::sort(chunks.begin(), chunks.end());
    uint32_t at = from / stride * stride;
    for (const auto& c : chunks) {
        if (c.first != at || c.second <= c.first || c.second - c.first > 32) {
            std::printf("FAIL n=%u warps=%u: chunk [%u, %u) after ray %u\n", n, warps, c.first, c.second, at);
            return 1;
        }
        at = c.second;
    }
    if (at != n) {
        std::printf("FAIL n=%u warps=%u: rays %u.. in no chunk\n", n, warps, at);
        return 1;
    }
    return 0;
}

int main() {
    int fails = 0;
    for (const uint32_t warps : {1u, 7u, 1216u, 5472u}) {
        const uint32_t far = 0xFFFFFFFFu - 20u * warps * 32u;
        for (uint32_t d = 0; d < 70; d++) {
            fails += check(warps * 32 * 3 + d, warps, 0);
            fails += check(0xFFFFFFFFu - d, warps, far);
        }
        for (const uint32_t n : {1u, 31u, 32u, 33u}) fails += check(n, warps, 0);
    }
    std::printf("%s: %d failures\n", fails ? "FAIL" : "ok", fails);
    return fails ? 1 : 0;
}

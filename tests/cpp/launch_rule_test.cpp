// launch_rule_test.cpp - the rules that pick the kernel, the claim size and the rays per warp of a
// launch, on the host: links libvrt.so and calls its planner (tile_launch, far_launch,
// resolve_launch_config, plan_views), and launch_rules.h.  Prints FAIL lines and exits non-zero on a mismatch.
#include <cstdio>
#include <vector>

#include "batch_internal.h"
#include "launch_rules.h"

using namespace vrt;

static int fails = 0;
#define CHECK(c)                                                          \
    do {                                                                  \
        if (!(c)) {                                                       \
            std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c);       \
            fails++;                                                      \
        }                                                                 \
    } while (0)

static vrt_view make(uint32_t w, uint32_t h, uint32_t bounces = 0, bool sun = false, int32_t wo = 0) {
    vrt_view v{};
    v.cam.width = w;
    v.cam.height = h;
    v.cam.d0[2] = 1.0f;
    v.cam.du[0] = 1.0f / w;
    v.cam.dv[1] = 1.0f / h;
    v.cam.world_origin[1] = wo;
    v.n_bounces = bounces;
    if (sun) {
        v.flags = VRT_VIEW_SHADOW;
        v.sun_dir[1] = 1.0f;
    }
    return v;
}

// chunk_tiles of a launch of `views` on `warps` warps, of which the caller set `chunk`
static uint32_t chunk(const std::vector<vrt_view>& views, uint64_t warps, uint32_t set = 0) {
    vrt_batch_config c{};
    normalize_batch_config(nullptr, c);
    c.chunk_tiles = set;
    resolve_launch_config(c, views.data(), (uint32_t)views.size(), warps);
    LaunchPlan plan;
    vrt_batch_config open{};
    normalize_batch_config(nullptr, open);
    open.chunk_tiles = set;
    CHECK(plan_views(views.data(), (uint32_t)views.size(), 1, open, plan, warps) == VRT_OK);
    CHECK(plan.cfg.chunk_tiles == c.chunk_tiles);
    CHECK(plan.tiles == tile_launch(views.data(), (uint32_t)views.size()));
    CHECK(plan.stall == stall_launch(views.data(), (uint32_t)views.size()));
    return c.chunk_tiles;
}

int main() {
    // the kernel: tile_kernel without bounces; not where a world origin is not near
    auto tiles = [](std::vector<vrt_view> v) { return tile_launch(v.data(), (uint32_t)v.size()); };
    auto far = [](std::vector<vrt_view> v) { return far_launch(v.data(), (uint32_t)v.size()); };
    CHECK(tiles({make(64, 64), make(8, 8, 0, true)}));
    CHECK(!tiles({make(64, 64), make(8, 8, 1)}));
    CHECK(!tiles({make(64, 64), make(8, 8, 2, true)}));
    const int32_t near = 1 << 22;
    for (const int32_t wo : {near - 1, -near}) CHECK(tiles({make(8, 8, 0, false, wo)}) && !far({make(8, 8, 0, false, wo)}));
    for (const int32_t wo : {near, -near - 1, 1 << 30, -(1 << 30)}) {
        CHECK(!tiles({make(64, 64), make(8, 8, 0, false, wo)}));
        CHECK(far({make(64, 64), make(8, 8, 3, true, wo)}));
    }
    // the test for rays that stand still: far views, and GLSL cameras with a whole coordinate
    auto stall = [](float x, uint32_t flags, int32_t wo = 0) {
        vrt_view v = make(8, 8, 2, false, wo);
        for (float& o : v.cam.origin) o = 0.25f;
        v.cam.origin[1] = x;
        v.flags |= flags;
        return stall_launch(&v, 1);
    };
    const uint32_t glsl = VRT_VIEW_GLSL, aniso = VRT_VIEW_GLSL | VRT_VIEW_GLSL_ANISO;
    for (const uint32_t f : {glsl, aniso}) {
        for (const float x : {0.0f, -0.0f, 3.0f, -16.0f, 1e9f}) CHECK(stall(x, f) && !stall(x, 0));
        for (const float x : {0.5f, 63.999f, -1e-6f}) CHECK(!stall(x, f) && stall(x, f, near));
    }
    CHECK(stall(0.5f, 0, near) && !stall(0.5f, 0, near - 1));

    // claims of tile_kernel, left open: at most 2 tiles, 1 with sun rays below 64 tiles a warp
    const uint64_t warps = 100;
    const std::vector<vrt_view> few = {make(640, 640)};              // 6,400 tiles: 64 a warp
    const std::vector<vrt_view> fewer = {make(640, 632)};            // 6,320 tiles
    CHECK(chunk(few, warps) == 2 && chunk(fewer, warps) == 2);
    CHECK(chunk({make(640, 640, 0, true)}, warps) == 2);
    CHECK(chunk({make(640, 632, 0, true)}, warps) == 1);
    CHECK(chunk({make(640, 320), make(640, 312, 0, true)}, warps) == 1);   // some view has sun rays
    CHECK(chunk({make(64, 64)}, warps) == 1);                        // 64 tiles
    CHECK(chunk({make(1592, 64)}, warps) == 1 && chunk({make(1600, 64)}, warps) == 2);  // 16 a warp: 8 claims of 2
    CHECK(chunk({make(1600, 1600)}, warps) == 2);
    CHECK(chunk({make(64, 64)}, 0) == 1 && chunk({make(64, 64, 0, true)}, 0) == 1);  // warps not known
    // with bounces one tile; values a caller set are kept
    CHECK(chunk({make(1600, 1600, 2)}, warps) == 1);
    for (const uint32_t set : {1u, 3u, 64u})
        CHECK(chunk(few, warps, set) == set && chunk({make(64, 64, 0, true)}, warps, set) == set &&
              chunk({make(64, 64, 2)}, warps, set) == set);
    // far views run on the persistent kernel: about eight claims a warp, 1 to 16 tiles
    CHECK(chunk({make(1600, 1600, 0, false, near)}, warps) == auto_chunk_tiles(40000, warps));
    CHECK(chunk({make(64, 64, 0, true, near)}, warps) == 1);

    // rays per warp and claims per tile, on 152 SMs and on half of them
    for (const uint32_t sms : {152u, 76u}) {
        const uint32_t w = 16 * sms;
        for (uint32_t l = 2; l < 5; l++) {
            const uint64_t most = ((uint64_t)w << l) + (1u << l) - 1;  // `w` warps of 2^l rays and a remainder below one
            CHECK(thin_lanes_log2(most, sms) == l && thin_lanes_log2(most + 1, sms) == l + 1);
        }
        CHECK(thin_lanes_log2(1, sms) == 2 && thin_lanes_log2(1ull << 32, sms) == 5);
        for (const bool bounces : {false, true}) {
            for (uint32_t k = 2; k <= 4; k++) CHECK(claim_split_log2(w >> k, bounces, sms) == k);
            CHECK(claim_split_log2(1, bounces, sms) == 4 && claim_split_log2((w >> 4) + 1, bounces, sms) == 3);
            CHECK(claim_split_log2((w >> 2) + 1, bounces, sms) == 1);
            CHECK(claim_split_log2(48 * sms, bounces, sms) == 1);
            CHECK(claim_split_log2(48 * sms + 1, bounces, sms) == (bounces ? 1 : 0));
        }
        CHECK(claim_split_log2(1u << 30, true, sms) == 1 && claim_split_log2((1u << 30) + 1, true, sms) == 0);
    }

    std::printf("%s: %d failures\n", fails ? "FAIL" : "ok", fails);
    return fails ? 1 : 0;
}

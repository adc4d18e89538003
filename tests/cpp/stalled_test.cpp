// stalled_test.cpp - dda_trace (trace_core.cuh), which ends rays that stand still between slices
// of steps, on the host, over the same files as device_logic_test.cpp:
//
//   stalled_test <world.bin> <rays.bin> <out.bin> <max_iters> <wox> <woy> <woz> <glsl> <coarse> <aniso>
#define main device_logic_main
#include "device_logic_test.cpp"
#undef main

template <typename T>
static std::vector<T> read_all(FILE* f, size_t n) {
    std::vector<T> v(n);
    if (std::fread(v.data(), sizeof(T), n, f) != n) std::exit(5);
    return v;
}

template <bool kGlsl>
static uint4 trace(const DevWorld& w, const vrt_ray& q, const int32_t wo[3], uint32_t iters, bool coarse, bool aniso) {
    RayState s;
    ray_start<kGlsl>(s, clip_box(w, wo), q.origin[0], q.origin[1], q.origin[2], q.dir[0], q.dir[1], q.dir[2], wo[0], wo[1],
                     wo[2], coarse);
    uint32_t i = 0;
    const bool hit = dda_trace<kGlsl, !kGlsl>(s, w, wo[0], wo[1], wo[2], coarse, coarse, aniso, i, iters,
                                              kGlsl && !coarse ? 8 : 16) == kStepHit;
    return pack_state<kGlsl>(s, hit_material(s, w.payload, hit), hit, i, q.tag);
}

int main(int argc, char** argv) {
    if (argc < 11) return 2;
    fill_forward_lut_entries(0, 1);
    FILE* f = std::fopen(argv[1], "rb");
    if (!f) return 3;
    const auto dims = read_all<uint32_t>(f, 4);
    const auto bricks = read_all<uint32_t>(f, (size_t)dims[0] * dims[1] * dims[2] * 64);
    const auto codes = read_all<uint8_t>(f, (size_t)dims[3] * 512), payload = read_all<uint8_t>(f, (size_t)dims[3] * 512);
    const auto cells = read_all<uint64_t>(f, (size_t)dims[3] * 8);
    std::fclose(f);
    DevWorld w{};
    w.bricks = bricks.data();
    w.codes = codes.data();
    w.payload = payload.data();
    w.cells = cells.data();
    w.bsx = dims[0] * 4;
    w.bsxz = dims[0] * 4 * dims[2] * 4;
    w.size_x = dims[0] * 32;
    w.size_y = dims[1] * 32;
    w.size_z = dims[2] * 32;
    const uint32_t iters = (uint32_t)std::atoi(argv[4]);
    const int32_t wo[3] = {std::atoi(argv[5]), std::atoi(argv[6]), std::atoi(argv[7])};
    const bool glsl = std::atoi(argv[8]) != 0, coarse = std::atoi(argv[9]) != 0, aniso = std::atoi(argv[10]) != 0;
    f = std::fopen(argv[2], "rb");
    FILE* o = std::fopen(argv[3], "wb");
    if (!f || !o) return 8;
    vrt_ray q;
    while (std::fread(&q, sizeof(q), 1, f) == 1) {
        const uint4 r = glsl ? trace<true>(w, q, wo, iters, coarse, aniso) : trace<false>(w, q, wo, iters, false, false);
        std::fwrite(&r, sizeof(r), 1, o);
    }
    std::fclose(o);
    return 0;
}

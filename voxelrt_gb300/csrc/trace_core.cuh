// trace_core.cuh - per-ray brickmap traversal on the device.
//
// One thread walks one ray through brick table -> voxel code -> voxel, the
// loop of RayCast/GetStepPos (src/VoxelRT/CpuRenderer.cpp:135-224) with the entry
// clip of clipRayToAABB (src/VoxelRT/Shaders/VoxelTraversal.glsl:133-145).
// Every float op is an explicitly rounded intrinsic (__fadd_rn, __fmul_rn,
// __fdiv_rn, __frcp_rn, __fsqrt_rn) in the reference's source order, so results do not
// depend on -fmad; min/max use the x86 minps/maxps NaN rule and floor->int uses
// the x86 out-of-range value INT32_MIN (SIMD_AVX512.h:109,123).
#pragma once

#include <cstdint>

#include "vrt_internal.h"

namespace vrt {

__device__ __forceinline__ float min_x86(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float max_x86(float a, float b) { return a > b ? a : b; }

// floor to int; NaN and out-of-range give INT32_MIN as cvtps2dq does.
__device__ __forceinline__ int32_t floor2i(float x) {
    return (x >= -2147483648.0f && x < 2147483648.0f) ? __float2int_rd(x) : INT32_MIN;
}
__device__ __forceinline__ int32_t wadd(int32_t a, int32_t b) { return (int32_t)((uint32_t)a + (uint32_t)b); }
__device__ __forceinline__ int32_t wsub(int32_t a, int32_t b) { return (int32_t)((uint32_t)a - (uint32_t)b); }

// a + b rounded down.
__device__ __forceinline__ float add_rd(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rd(a, b);
#else
    // f - b is exact in double here (f and b are close, or f is an infinity or NaN)
    float f = (float)((double)a + (double)b);
    if ((double)f - (double)b > (double)a) {
        uint32_t u = __float_as_uint(f);
        u = f > 0.0f ? u - 1u : (f < 0.0f ? u + 1u : 0x80000001u);
        f = __uint_as_float(u);
    }
    return f;
#endif
}

// Two float adds in one instruction (sm_100 and later), each rounded as its scalar form: the step
// loop is bound by instruction issue, and x and y take the same operations. 1080p frame with
// a shadow ray 126.7 -> 121.8 us, 1080p x 8 views 754 -> 742, 64 mixed views 679 -> 671, an
// anisotropic path batch 710 -> 694. The products stay scalar: with a packed multiply that feeds a
// packed add the records differ from the oracle's, as a fused multiply-add's would.
struct F2 {
    float x, y;
};
#ifdef __CUDA_ARCH__
#define VRT_F2_ADD(name, op)                                                                 \
    __device__ __forceinline__ F2 name(F2 a, F2 b) {                                         \
        F2 r;                                                                                \
        asm("{\n.reg .b64 a, b, r;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\n" op         \
            " r, a, b;\nmov.b64 {%0, %1}, r;\n}"                                             \
            : "=f"(r.x), "=f"(r.y)                                                           \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                       \
        return r;                                                                            \
    }
VRT_F2_ADD(add2, "add.rn.f32x2")
VRT_F2_ADD(add2_rd, "add.rm.f32x2")
#undef VRT_F2_ADD
#else
__device__ __forceinline__ F2 add2(F2 a, F2 b) { return F2{__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)}; }
__device__ __forceinline__ F2 add2_rd(F2 a, F2 b) { return F2{add_rd(a.x, b.x), add_rd(a.y, b.y)}; }
#endif

// Voxel coordinates as floats with an integer part in the low bits.  kVoxelBias is the
// bit pattern of M = 1.5 * 2^23, where one ulp is 1: for an integer |n| < 2^22 the float
// M + n has the bits kVoxelBias + n.  With a near world origin the float K = M + worldOrigin
// is exact, and add_rd(pos, K) is M + worldOrigin + floor(pos): one add on the FMA pipe takes
// the place of a conversion (on a quarter-rate unit, the longest latency in the step's chain)
// and of the add of worldOrigin.  A position out of the grid, an infinity or NaN among them,
// gives bits below kVoxelBias or at least the grid's size above it (unsigned).  Back in the ray
// frame, the float minus K is exactly voxel - worldOrigin.
constexpr uint32_t kVoxelBias = 0x4B400000u;
// K of an axis
__device__ __forceinline__ float voxel_frame(int32_t wo) { return __uint_as_float(kVoxelBias + (uint32_t)wo); }

// v - worldOrigin (wrapping), the ray-frame coordinate of a voxel
__device__ __forceinline__ float rel_voxel(int32_t v, int32_t wo) {
    return __int2float_rn(wsub(v, wo));
}

struct TraceResult {
    float cx, cy, cz;  // final position (HitResult.Pos)
    float sx, sy, sz;  // final side distances
    float tb;          // GLSL mode: biased tmin of the last step (hit.dist)
    uint32_t voxel;    // of a hit, as the record packs it
    uint32_t steps;
    uint32_t material;
    bool hit;
};

struct TraceCounters {
    uint32_t step_calls;
    uint32_t occ_fetches;
};

// 1/sqrt(l2) for the normalisation of camera rays: the integer first estimate
// 0x5F3759DF - (bits(l2) >> 1) (C. Lomont, "Fast Inverse Square Root", 2003), then
// three Newton steps r <- r * (1.5 - (l2/2) * r*r), each one exactly rounded multiply,
// one fused multiply-add and one multiply, so any IEEE machine gets the same bits.
// For l2 in [2^-126, 2^126] the result is within 2.5 ulp of 1/sqrt(l2); the reference
// normalises with a 14-bit hardware estimate (SIMD.h normalize, rsqrt14).
__device__ __forceinline__ float camera_rsqrt(float l2) {
    const float h = __fmul_rn(0.5f, l2);
    float r = __uint_as_float(0x5F3759DFu - (__float_as_uint(l2) >> 1));
#pragma unroll
    for (int i = 0; i < 3; i++) r = __fmul_rn(r, __fmaf_rn(-h, __fmul_rn(r, r), 1.5f));
    return r;
}

// Ray entry point of a camera pixel (the ray generation of vrt_camera) from the
// camera's d0, du, dv vectors.
__device__ __forceinline__ void camera_ray(const float* d0, const float* du, const float* dv, uint32_t px,
                                           uint32_t py, float& dx, float& dy, float& dz) {
    float u = __fadd_rn(__uint2float_rn(px), 0.5f);
    float v = __fadd_rn(__uint2float_rn(py), 0.5f);
    float x = __fadd_rn(__fadd_rn(d0[0], __fmul_rn(u, du[0])), __fmul_rn(v, dv[0]));
    float y = __fadd_rn(__fadd_rn(d0[1], __fmul_rn(u, du[1])), __fmul_rn(v, dv[1]));
    float z = __fadd_rn(__fadd_rn(d0[2], __fmul_rn(u, du[2])), __fmul_rn(v, dv[2]));
    const float r = camera_rsqrt(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
    dx = __fmul_rn(x, r);
    dy = __fmul_rn(y, r);
    dz = __fmul_rn(z, r);
}
__device__ __forceinline__ void camera_ray(const vrt_camera& cam, uint32_t px, uint32_t py, float& dx,
                                           float& dy, float& dz) {
    camera_ray(cam.d0, cam.du, cam.dv, px, py, dx, dy, dz);
}

// Per-ray traversal state: RayCast's loop-carried values (CpuRenderer.cpp:173-184).
struct RayState {
    float ox, oy, oz, dx, dy, dz;
    float ix, iy, iz;     // invDir
    float tsx, tsy, tsz;  // tStart
    float cx, cy, cz;     // currPos
    float sx, sy, sz;     // sideDist
    float tb;             // GLSL mode: biased tmin of the last step
    bool fast;            // the ray takes the fast step (ray_init)
    int32_t gx, gy, gz;   // -1 where dir < 0, else 0 (cell alignment side)
    // A hit ends the use of tStart: the step that hits leaves the voxel (as the record packs
    // it) and the brick's slot there, so a lane waiting for its retirement holds no more.
    __device__ __forceinline__ void set_hit(uint32_t x, uint32_t y, uint32_t z, uint32_t slot) {
        tsx = __uint_as_float(x | y << 11 | z << 21);
        tsy = __uint_as_float(slot);
    }
    __device__ __forceinline__ uint32_t hit_voxel() const { return __float_as_uint(tsx); }
    __device__ __forceinline__ size_t hit_byte() const {  // of the payload
        const uint32_t v = __float_as_uint(tsx);
        return (size_t)__float_as_uint(tsy) * 512 + ((v & 7u) | ((v >> 21) & 7u) << 3 | ((v >> 11) & 7u) << 6);
    }
};

// A ray takes the fast step (ray_step<.., true>) when no NaN or infinity can occur in its side
// distances and voxels of the grid have their biased form:
// - -2^22 <= worldOrigin < 2^22 (a near one), so K is exact;
// - |origin| < 2^30 and |1/dir| < 2^95: |tStart| and |(voxel - worldOrigin) * invDir| stay below
//   2^126, so side distances and t are finite, and the position o + t*d is finite or an
//   infinity (never NaN) that leaves the grid.
constexpr int32_t kNearWorldOrigin = 1 << 22;
constexpr float kFastOrigin = 0x1p30f, kFastInvDir = 0x1p95f;
VRT_HD inline bool near_origin(const int32_t wo[3]) {
    bool near = true;
    for (int c = 0; c < 3; c++) near &= (uint32_t)wo[c] + (uint32_t)kNearWorldOrigin < 2u * (uint32_t)kNearWorldOrigin;
    return near;
}

// The clip box [1 - worldOrigin, size - 1 - worldOrigin] (VoxelTraversal.glsl:166) of a world
// origin, and whether that is near: the same for every ray of a view or cast.
struct ClipBox {
    float lo[3], hi[3];
    uint32_t near;
};
VRT_HD inline ClipBox clip_box(const DevWorld& w, const int32_t wo[3]) {
    const uint32_t size[3] = {w.size_x, w.size_y, w.size_z};
    ClipBox b;
    for (int c = 0; c < 3; c++) {
        b.lo[c] = (float)(1 - wo[c]);
        b.hi[c] = ((float)size[c] - (float)wo[c]) - 1.0f;
    }
    b.near = near_origin(wo) ? 1u : 0u;
    return b;
}
// The box holds the origin strictly inside, and the world origin is near: a ray's start then
// needs neither the slab test nor the bounds of the origin.  Camera rays of a view share
// their origin, so this is evaluated once per view, or per claimed chunk.
VRT_HD inline bool origin_inside_near(const ClipBox& b, float ox, float oy, float oz) {
    return b.near && b.lo[0] < ox && ox < b.hi[0] && b.lo[1] < oy && oy < b.hi[1] && b.lo[2] < oz && oz < b.hi[2];
}
// What every start sets: origin, direction, invDir, tStart, the alignment sides.
__device__ __forceinline__ void ray_set(RayState& s, float ox, float oy, float oz, float dx, float dy, float dz) {
    s.ox = s.cx = ox;
    s.oy = s.cy = oy;
    s.oz = s.cz = oz;
    s.dx = dx;
    s.dy = dy;
    s.dz = dz;
    // correctly rounded 1/dir, the same value as the IEEE division 1.0f / dir
    s.ix = __frcp_rn(dx);
    s.iy = __frcp_rn(dy);
    s.iz = __frcp_rn(dz);
    s.tsx = __fmul_rn(__fsub_rn(dx < 0.0f ? 0.0f : 1.0f, ox), s.ix);
    s.tsy = __fmul_rn(__fsub_rn(dy < 0.0f ? 0.0f : 1.0f, oy), s.iy);
    s.tsz = __fmul_rn(__fsub_rn(dz < 0.0f ? 0.0f : 1.0f, oz), s.iz);
    s.gx = dx < 0.0f ? -1 : 0;
    s.gy = dy < 0.0f ? -1 : 0;
    s.gz = dz < 0.0f ? -1 : 0;
    s.sx = s.sy = s.sz = 0.0f;
    s.fast = fabsf(s.ix) < kFastInvDir && fabsf(s.iy) < kFastInvDir && fabsf(s.iz) < kFastInvDir;
}

// Start of any ray, with the clipped start position (VoxelTraversal.glsl:133-145,163-167).  An
// origin inside and near never clips: per axis l - o < 0 < h - o, so min(t1, t2) is negative
// (or -inf, or NaN when dir is NaN, which minps/maxps drop) and tmin <= 0 on every path; for
// one known to be, ray_set is the whole start.
__device__ __forceinline__ void ray_init(RayState& s, const ClipBox& b, float ox, float oy, float oz, float dx,
                                         float dy, float dz) {
    ray_set(s, ox, oy, oz, dx, dy, dz);
    if (origin_inside_near(b, ox, oy, oz)) return;
    const float t1x = __fmul_rn(__fsub_rn(b.lo[0], ox), s.ix), t2x = __fmul_rn(__fsub_rn(b.hi[0], ox), s.ix);
    const float t1y = __fmul_rn(__fsub_rn(b.lo[1], oy), s.iy), t2y = __fmul_rn(__fsub_rn(b.hi[1], oy), s.iy);
    const float t1z = __fmul_rn(__fsub_rn(b.lo[2], oz), s.iz), t2z = __fmul_rn(__fsub_rn(b.hi[2], oz), s.iz);
    const float tmin = max_x86(min_x86(t1x, t2x), max_x86(min_x86(t1y, t2y), min_x86(t1z, t2z)));
    const float tmax = min_x86(max_x86(t1x, t2x), min_x86(max_x86(t1y, t2y), max_x86(t1z, t2z)));
    if (tmin > 0.0f && tmin < tmax) {
        s.cx = __fadd_rn(ox, __fmul_rn(dx, tmin));
        s.cy = __fadd_rn(oy, __fmul_rn(dy, tmin));
        s.cz = __fadd_rn(oz, __fmul_rn(dz, tmin));
    }
    s.fast = s.fast && b.near && fabsf(ox) < kFastOrigin && fabsf(oy) < kFastOrigin && fabsf(oz) < kFastOrigin;
}

// The position at distance t.
__device__ __forceinline__ void set_position(RayState& s, float t) {
    const F2 c = add2(F2{s.ox, s.oy}, F2{__fmul_rn(t, s.dx), __fmul_rn(t, s.dy)});
    s.cx = c.x;
    s.cy = c.y;
    s.cz = __fadd_rn(s.oz, __fmul_rn(t, s.dz));
}

// GLSL mode: the step's distance and position from its side distances.  tmin + 5 ulp as
// an integer add on the bits; a NaN tmin stays NaN (its bit pattern differs between
// platforms: the GPU's 0x7FFFFFFF would wrap to a denormal).  A rayCastCoarse ray takes
// tmin + 0.001 (VoxelTraversal.glsl:213).  Kept as the hit distance, so min keeps the minps
// rule.
template <bool kFast>
__device__ __forceinline__ void glsl_advance(RayState& s, bool coarse_ray) {
    const float m = min_x86(min_x86(s.sx, s.sy), s.sz);
    const float t = coarse_ray ? __fadd_rn(m, 0.001f) : (!kFast && m != m) ? m : __uint_as_float(__float_as_uint(m) + 5u);
    s.tb = t;
    set_position(s, t);
}

// GLSL mode (VoxelTraversal.glsl rayCast): the start voxel worldOrigin + floor(start), and
// the side distances and position that iteration 0 takes from it (:164-174), so that a step
// of either mode begins with its position and ends with the next one.
// coarse_origin (GLSL mode, a rayCastCoarse ray): the clipped start replaces the origin,
// so tStart, positions and the hit distance count from it (VoxelTraversal.glsl:207-210);
// rayCast keeps the origin and starts from the clipped voxel only (:162-167).  Without
// a clip the start is the origin and nothing changes.
template <bool kGlsl>
__device__ __forceinline__ void glsl_start(RayState& s, int32_t wox, int32_t woy, int32_t woz, bool coarse_origin) {
    if (!kGlsl) return;
    if (coarse_origin) {
        s.ox = s.cx;
        s.oy = s.cy;
        s.oz = s.cz;
        s.tsx = __fmul_rn(__fsub_rn(s.dx < 0.0f ? 0.0f : 1.0f, s.ox), s.ix);
        s.tsy = __fmul_rn(__fsub_rn(s.dy < 0.0f ? 0.0f : 1.0f, s.oy), s.iy);
        s.tsz = __fmul_rn(__fsub_rn(s.dz < 0.0f ? 0.0f : 1.0f, s.oz), s.iz);
    }
    // (voxel - worldOrigin in wrapping arithmetic, where the start voxel saturated)
    s.sx = __fadd_rn(s.tsx, __fmul_rn(rel_voxel(wadd(wox, floor2i(s.cx)), wox), s.ix));
    s.sy = __fadd_rn(s.tsy, __fmul_rn(rel_voxel(wadd(woy, floor2i(s.cy)), woy), s.iy));
    s.sz = __fadd_rn(s.tsz, __fmul_rn(rel_voxel(wadd(woz, floor2i(s.cz)), woz), s.iz));
    glsl_advance<false>(s, coarse_origin);
}

// A ray's start, and that of a ray whose origin is inside and near (origin_inside_near).
template <bool kGlsl>
__device__ __forceinline__ void ray_start(RayState& s, const ClipBox& b, float ox, float oy, float oz, float dx,
                                          float dy, float dz, int32_t wox, int32_t woy, int32_t woz,
                                          bool coarse_origin = false) {
    ray_init(s, b, ox, oy, oz, dx, dy, dz);
    glsl_start<kGlsl>(s, wox, woy, woz, coarse_origin);
}
template <bool kGlsl>
__device__ __forceinline__ void ray_start_inside(RayState& s, float ox, float oy, float oz, float dx,
                                                 float dy, float dz, int32_t wox, int32_t woy, int32_t woz) {
    ray_set(s, ox, oy, oz, dx, dy, dz);
    glsl_start<kGlsl>(s, wox, woy, woz, false);
}

enum : uint32_t { kStepContinue = 0, kStepHit = 1, kStepOut = 2 };

// Anisotropic LODs: RayCellInteractionMaskLUT (GpuRenderer.cpp:193-210) in shared
// memory, entry idx + 64 * octant (octant = (dx >= 0) | (dy >= 0) << 1 | (dz >= 0) << 2),
// [0] the forward box of cell idx and [1] its part inside idx's aligned 2^3 block, so
// that getIsotropicLod of the masked mask (VoxelTraversal.glsl:24-34) is two tests.
// Every kernel that traces with anisotropic LODs fills it first (fill_forward_lut).
#if defined(__CUDACC__)
static __shared__ uint64_t s_forward_lut[2][512];
#else
inline uint64_t s_forward_lut[2][512];
#endif

__device__ __forceinline__ void fill_forward_lut_entries(uint32_t first, uint32_t step) {
    for (uint32_t i = first; i < 512; i += step) {
        const uint32_t idx = i & 63u, o = i >> 6;
        const uint64_t f = forward_cells(idx, (o & 1u) ? 0 : -1, (o & 2u) ? 0 : -1, (o & 4u) ? 0 : -1);
        s_forward_lut[0][i] = f;
        s_forward_lut[1][i] = f & (0x330033ull << (idx & 0x2Au));
    }
}

#if defined(__CUDACC__)
// all threads of the block, before any of them returns
__device__ __forceinline__ void fill_forward_lut() {
    fill_forward_lut_entries(threadIdx.x + threadIdx.y * blockDim.x, blockDim.x * blockDim.y);
    __syncthreads();
}
#endif

// GLSL mode: rayCastCoarse (VoxelTraversal.glsl:206-240), the GPU renderer's shadow and
// bounce rays (VoxelRender.comp:56,74,81): kCoarseRay for every step of such a ray,
// kCoarseNow from its iteration 31 on (`coarse = i > 30`, :218).
enum : uint32_t { kCoarseRay = 1, kCoarseNow = 2 };
constexpr uint32_t kCoarseFrom = 31, kCoarseMaxIters = 96;
__device__ __forceinline__ uint32_t coarse_bits(bool coarse_ray, uint32_t i) {
    return coarse_ray ? (kCoarseRay | (i >= kCoarseFrom ? kCoarseNow : 0u)) : 0u;
}

// The end of a step: from the voxel (of a fast ray in its biased form) and the alignment
// mask of its cell to the cell's side distances, tmin and the next position.
template <bool kFast, bool kGlsl, bool kCoarse>
__device__ __forceinline__ void step_on(RayState& s, uint32_t vx, uint32_t vy, uint32_t vz, uint32_t m, int32_t wox,
                                        int32_t woy, int32_t woz, uint32_t coarse) {
    // dir < 0 ? pos & ~m : pos | m, as (pos | m) ^ (g & m) with g = -1 for dir < 0
    vx = (vx | m) ^ ((uint32_t)s.gx & m);
    vy = (vy | m) ^ ((uint32_t)s.gy & m);
    vz = (vz | m) ^ ((uint32_t)s.gz & m);
    if (kFast) {
        const F2 f = add2(F2{__uint_as_float(vx), __uint_as_float(vy)}, F2{-voxel_frame(wox), -voxel_frame(woy)});
        const float fz = __fsub_rn(__uint_as_float(vz), voxel_frame(woz));
        const F2 d = add2(F2{s.tsx, s.tsy}, F2{__fmul_rn(f.x, s.ix), __fmul_rn(f.y, s.iy)});
        s.sx = d.x;
        s.sy = d.y;
        s.sz = __fadd_rn(s.tsz, __fmul_rn(fz, s.iz));
    } else {
        s.sx = __fadd_rn(s.tsx, __fmul_rn(rel_voxel((int32_t)vx, wox), s.ix));
        s.sy = __fadd_rn(s.tsy, __fmul_rn(rel_voxel((int32_t)vy, woy), s.iy));
        s.sz = __fadd_rn(s.tsz, __fmul_rn(rel_voxel((int32_t)vz, woz), s.iz));
    }
    if (kGlsl) {
        glsl_advance<kFast>(s, kCoarse && (coarse & kCoarseRay) != 0);
    } else {
        const float t = kFast ? __fadd_rn(fminf(fminf(s.sx, s.sy), s.sz), 0.001f)
                              : __fadd_rn(min_x86(min_x86(s.sx, s.sy), s.sz), 0.001f);
        set_position(s, t);
    }
}

// One iteration of RayCast (CpuRenderer.cpp:186-201) with GetStepPos (:135-171): the voxel
// of the current position, its bounds and table entries, then the side distances of the cell
// reached, tmin and the next position.
// kFast: the ray passed the bounds of ray_init, so no NaN can occur and voxels are kept in the
// biased form of kVoxelBias; min uses fminf, which equals the minps rule on non-NaN operands
// up to the sign of a zero result, which the +0.001 bias removes.
// kGlsl: rayCast (VoxelTraversal.glsl:170-199), whose iteration takes its position first
// (ray_start has iteration 0's): bounds, then getStepPos (:100-131), whose empty sectors take
// the 4th-level mask from the brick table.  kCoarse (with kGlsl): the step may belong to a
// rayCastCoarse ray, as `coarse` (coarse_bits) says: from iteration 31 an empty voxel whose
// 4^3 cell holds a solid voxel stops the ray at the cell's first solid voxel in mask order
// (getStepPos with coarse, :125-128, and findAnyOccupiedPos, :41-53).  Without kCoarse
// `coarse` is 0.
// kAniso (with kGlsl): anisotropic LODs (u_UseAnisotropicLods, :116-121): the mask of
// the current level (cell, sector or sector group, read raw instead of through the
// precomputed codes) is restricted to the cells ahead of the ray before its LOD is taken.
// kFlat (not with kAniso): no branch on what the brick is.  A position outside reads no entry
// and takes kOutside, whose masks are the solid code, so one test ends the ray either way,
// and an allocated brick's code is a predicated load.  Fewer branches, more instructions for
// an empty brick: for rays that diverge in any case (bounces of two 720p views: 423 -> 409 us;
// 4.2 M random rays: 252 -> 248 us, 16,000: 20.2 -> 18.7 us); camera rays over terrain lose (six
// 1080p views with sun rays 779 -> 816 us).
constexpr uint32_t kOutside = kBrickEmpty | kCodeSolid | kCodeSolid << 8;
template <bool kCount, bool kFast, bool kGlsl, bool kCoarse, bool kAniso, bool kFlat>
__device__ __forceinline__ uint32_t ray_step(RayState& s, const DevWorld& w, int32_t wox, int32_t woy, int32_t woz,
                                             TraceCounters& cnt, uint32_t coarse = 0) {
    uint32_t vx, vy, vz;  // the voxel; of a fast ray its biased form
    constexpr uint32_t kBias = kFast ? kVoxelBias : 0u;
    if (kFast) {
        const F2 r = add2_rd(F2{s.cx, s.cy}, F2{voxel_frame(wox), voxel_frame(woy)});
        vx = __float_as_uint(r.x);
        vy = __float_as_uint(r.y);
        vz = __float_as_uint(add_rd(s.cz, voxel_frame(woz)));
    } else {
        // floor2i: a NaN coordinate converts to INT32_MIN on x86 and leaves the grid;
        // cvt.rmi saturates infinities and out-of-range values, which leave the grid
        // too (|world origin| <= 2^30 is enforced at the API), so only NaN needs a test
        // and one NaN among the three shows in their sum.
        const float nan_probe = __fadd_rn(__fadd_rn(s.cx, s.cy), s.cz);
        if (nan_probe != nan_probe) return kStepOut;
        vx = (uint32_t)wadd(__float2int_rd(s.cx), wox);
        vy = (uint32_t)wadd(__float2int_rd(s.cy), woy);
        vz = (uint32_t)wadd(__float2int_rd(s.cz), woz);
    }
    const uint32_t ux = vx - kBias, uy = vy - kBias, uz = vz - kBias;
    const bool in = ux < w.size_x && uy < w.size_y && uz < w.size_z;
    // (the sum in 32 bits: added to the pointer term by term 44 M camera rays took 698 us against 679)
    const uint32_t ei = (uy >> 3) * w.bsxz + ((uz >> 3) * w.bsx + (ux >> 3));
    const uint32_t vi = (ux & 7u) | (uz & 7u) << 3 | (uy & 7u) << 6;  // voxel in brick x | z<<3 | y<<6
    // The brick table holds the slot of an allocated brick, or for an empty one the
    // alignment mask of the level GetStepPos reaches from the sector mask
    // (3 + skip_levels).  An allocated brick's voxel code is kCodeSolid (the hit) or
    // the alignment mask of the skip level of the voxel's 4^3 cell; both replace the
    // two mask fetches of the reference with their precomputed outcome.
    uint32_t e, m;
    if (kAniso) {
        if (!in) return kStepOut;
        if (kCount) cnt.step_calls++;
        e = __ldg(w.bricks + ei);
        if (e < kBrickEmpty) {
            if (kCount) cnt.occ_fetches++;
            const uint32_t lx = ux & 7u, ly = uy & 7u, lz = uz & 7u;
            const uint64_t cm = __ldg(w.cells + (size_t)e * 8 + ((lx >> 2) | (lz >> 2) << 1 | (ly >> 2) << 2));
            const uint32_t idx = (lx & 3u) | (lz & 3u) << 2 | (ly & 3u) << 4;
            if ((cm >> idx) & 1u) {
                s.set_hit(ux, uy, uz, e);
                return kStepHit;
            }
            const uint32_t li = idx + 64u * ((uint32_t)(s.gx + 1) | (uint32_t)(s.gy + 1) << 1 | (uint32_t)(s.gz + 1) << 2);
            const uint64_t am = cm & s_forward_lut[0][li];
            if (kCoarse && (coarse & kCoarseNow) && am != 0) {
                // findAnyOccupiedPos on the masked cell mask: its lowest set bit
                const uint32_t j = (uint32_t)__ffsll((long long)am) - 1u;
                s.set_hit((ux & ~3u) | (j & 3u), (uy & ~3u) | (j >> 4), (uz & ~3u) | ((j >> 2) & 3u), e);
                return kStepHit;
            }
            m = am == 0 ? 3u : ((cm & s_forward_lut[1][li]) == 0 ? 1u : 0u);
        } else {
            // an empty brick: the sector mask (scale 8) or, in an empty sector, the
            // sector-group mask (scale 32) restricted to the ray's octant, whose skip level
            // the table entry carries per octant
            const uint32_t oct2 = ((uint32_t)(s.gx + 1) | (uint32_t)(s.gy + 1) << 1 | (uint32_t)(s.gz + 1) << 2) * 2u;
            const uint32_t skip = ((e >> (kAnisoShift + oct2)) & 3u) + ((e >> 4) & 2u);
            m = (8u << skip) - 1u;
        }
    } else if (kFlat) {
        e = kOutside;
        if (in) e = __ldg(w.bricks + ei);
        if (kCount && in) cnt.step_calls++;
        m = kGlsl ? (e >> 8) & 127u : e & 31u;
        if (e < kBrickEmpty) m = __ldg(w.codes + (size_t)e * 512 + vi);
        if (kCount && e < kBrickEmpty) cnt.occ_fetches++;
        if (m == kCodeSolid) {
            if (e == kOutside) return kStepOut;
            s.set_hit(ux, uy, uz, e);
            return kStepHit;
        }
    } else {
        if (!in) return kStepOut;
        if (kCount) cnt.step_calls++;
        e = __ldg(w.bricks + ei);
        if (e < kBrickEmpty) {
            if (kCount) cnt.occ_fetches++;
            m = __ldg(w.codes + (size_t)e * 512 + vi);
            if (m == kCodeSolid) {
                s.set_hit(ux, uy, uz, e);
                return kStepHit;
            }
        } else {
            m = kGlsl ? (e >> 8) & 127u : e & 31u;
        }
    }
    if (kGlsl && kCoarse && !kAniso && (coarse & kCoarseNow) && e < kBrickEmpty && m != 3u) {
        // the cell's mask is not empty (lod < 4): its first solid voxel, bit
        // x + z*4 + y*16 of the cell mask, is the hit (mask-order scan of the payload)
        const size_t cell = (size_t)e * 512 + ((ux & 4u) | (uz & 4u) << 3 | (uy & 4u) << 6);
        for (uint32_t j = 0; j < 64; j++) {
            if (__ldg(w.payload + cell + ((j & 3u) | ((j >> 2) & 3u) << 3 | (j >> 4) << 6))) {
                s.set_hit((ux & ~3u) | (j & 3u), (uy & ~3u) | (j >> 4), (uz & ~3u) | ((j >> 2) & 3u), e);
                return kStepHit;
            }
        }
    }
    step_on<kFast, kGlsl, kCoarse>(s, vx, vy, vz, m, wox, woy, woz, coarse);
    return kStepContinue;
}

// Steps k = k .. kmax-1 of a ray whose first step here is its iteration i0 + k, until
// one ends it (the returned status) or kmax is reached (kStepContinue).  The general step's loop
// follows the fast one, which it leaves in place: with a choice between the two a step took 59 warp
// instructions instead of 49 (smsp__inst_executed at caps of 1 and 5 steps).  A test of the distance
// against the grid's exit in place of the three bounds compares saved nothing, and lanes past the
// exit, stepping in the second loop, doubled the time of warps with stalled rays.
// coarse_ray: a rayCastCoarse ray (kCoarse only).
template <bool kCount, bool kGlsl, bool kCoarse, bool kAniso, bool kFlat>
__device__ __forceinline__ uint32_t dda_steps(RayState& s, const DevWorld& w, int32_t wox, int32_t woy, int32_t woz,
                                              TraceCounters& cnt, bool coarse_ray, uint32_t i0, uint32_t& k,
                                              uint32_t kmax) {
    uint32_t st = kStepContinue;
    const uint32_t kfast = s.fast ? kmax : 0u;
    while (k < kfast) {
        st = ray_step<kCount, true, kGlsl, kCoarse, kAniso, kFlat>(s, w, wox, woy, woz, cnt,
                                                            kCoarse ? coarse_bits(coarse_ray, i0 + k) : 0u);
        if (st != kStepContinue) return st;
        k++;
    }
    for (; k < kmax; k++) {
        st = ray_step<kCount, false, kGlsl, kCoarse, kAniso, false>(s, w, wox, woy, woz, cnt,
                                                             kCoarse ? coarse_bits(coarse_ray, i0 + k) : 0u);
        if (st != kStepContinue) break;
    }
    return st;
}

// dda_steps with the GLSL variants picked at run time: coarse (some ray of the caller's
// group may be a rayCastCoarse ray; coarse_ray says whether this one is) and aniso.
template <bool kCount, bool kGlsl, bool kFlat = false>
__device__ __forceinline__ uint32_t dda_steps_mode(RayState& s, const DevWorld& w, int32_t wox, int32_t woy,
                                                   int32_t woz, TraceCounters& cnt, bool coarse,
                                                   bool coarse_ray, bool aniso, uint32_t i0, uint32_t& k,
                                                   uint32_t kmax) {
    if constexpr (!kGlsl) {
        return dda_steps<kCount, false, false, false, kFlat>(s, w, wox, woy, woz, cnt, false, i0, k, kmax);
    } else {
        if (aniso)
            return coarse ? dda_steps<kCount, true, true, true, false>(s, w, wox, woy, woz, cnt, coarse_ray, i0, k, kmax)
                          : dda_steps<kCount, true, false, true, false>(s, w, wox, woy, woz, cnt, false, i0, k, kmax);
        return coarse ? dda_steps<kCount, true, true, false, kFlat>(s, w, wox, woy, woz, cnt, coarse_ray, i0, k, kmax)
                      : dda_steps<kCount, true, false, false, kFlat>(s, w, wox, woy, woz, cnt, false, i0, k, kmax);
    }
}

// Rays that stand still.  Where the bias of a step's distance (0.001, or 5 ulp in GLSL mode) is lost
// in the rounding of the position, a ray stays before the cell's face and repeats its step up
// to the iteration cap: an explicit ray has its origin in world coordinates, and of random rays
// through a 256-voxel terrain one in four stands still in GLSL mode (256 steps each) and one in 500
// in CPU mode.  A step is a function of the position, and the position of the distance alone, so a
// ray back at the distance it had some steps before repeats those steps, none of which ended
// it: its record is that of the cap.  (A distance of NaN equals none.)  Of a rayCastCoarse ray
// (coarse_ray) once its steps no longer depend on their number.
// Looked at between slices of steps: 2,000 random GLSL rays 49 -> 13 us, 2.5 M 653 -> 112, 2.5 M
// anisotropic 841 -> 128, 60,000 CPU rays in a mixed world 22.9 -> 12.1; 1 M CPU rays from 2^22 voxels
// off the world origin 290 -> 68.  The persistent kernel looks too (batch.cu), in launches of the GLSL
// modes, where a third of a camera's rays stand still when it lies in the plane of an empty brick's
// face, and of views whose world origin is not near, nearly all of whose rays do.  Other frames and batches look for none: the
// slices' loop cost them 2 to 8 %.
template <bool kGlsl>
__device__ __forceinline__ float last_t(const RayState& s) {
    return kGlsl ? s.tb : min_x86(min_x86(s.sx, s.sy), s.sz);
}
__device__ __forceinline__ float no_t() { return __uint_as_float(0x7FFFFFFFu); }  // equals no distance
// t0: last_t before iteration `first`, with one step or more since.
template <bool kGlsl>
__device__ __forceinline__ bool stalled(const RayState& s, float t0, bool coarse_ray, uint32_t first) {
    return last_t<kGlsl>(s) == t0 && (!kGlsl || !coarse_ray || first >= kCoarseFrom);
}

// dda_steps_mode from iteration i to the ray's end or `iters`, `slice` steps at a time.
template <bool kGlsl, bool kFlat>
__device__ __forceinline__ uint32_t dda_trace(RayState& s, const DevWorld& w, int32_t wox, int32_t woy, int32_t woz,
                                              bool coarse, bool coarse_ray, bool aniso, uint32_t& i, uint32_t iters,
                                              uint32_t slice) {
    TraceCounters cnt{0, 0};
    float t0 = no_t();
    for (;;) {
        const uint32_t first = i, lim = iters - i < slice ? iters : i + slice;
        const uint32_t st =
            dda_steps_mode<false, kGlsl, kFlat>(s, w, wox, woy, woz, cnt, coarse, coarse_ray, aniso, 0, i, lim);
        if (st != kStepContinue || i >= iters) return st;
        if (stalled<kGlsl>(s, t0, coarse_ray, first)) {
            i = iters;
            return st;
        }
        t0 = last_t<kGlsl>(s);
    }
}

// Voxel id of a hit (0 on a miss), read once its ray has ended.
__device__ __forceinline__ uint32_t hit_material(const RayState& s, const uint8_t* payload, bool hit) {
    return hit ? __ldg(payload + s.hit_byte()) : 0u;
}

// Whole RayCast (or rayCast / rayCastCoarse, kGlsl) for one ray.
template <bool kCount, bool kGlsl = false>
__device__ __forceinline__ void trace_ray(const DevWorld& w, float ox, float oy, float oz, float dx, float dy,
                                          float dz, int32_t wox, int32_t woy, int32_t woz, uint32_t max_iters,
                                          TraceResult& r, TraceCounters& cnt, bool coarse_ray = false,
                                          bool aniso = false) {
    RayState s;
    const int32_t wo[3] = {wox, woy, woz};
    ray_start<kGlsl>(s, clip_box(w, wo), ox, oy, oz, dx, dy, dz, wox, woy, woz, coarse_ray);
    uint32_t i = 0;
    uint32_t st = dda_steps_mode<kCount, kGlsl>(s, w, wox, woy, woz, cnt, coarse_ray, coarse_ray, aniso, 0, i,
                                                max_iters);
    if (max_iters == 0) st = kStepOut;
    r.cx = s.cx;
    r.cy = s.cy;
    r.cz = s.cz;
    r.sx = s.sx;
    r.sy = s.sy;
    r.sz = s.sz;
    r.tb = s.tb;
    r.voxel = s.hit_voxel();
    r.steps = i;  // == max_iters when the cap ran out
    r.hit = st == kStepHit && i < max_iters;
    r.material = hit_material(s, w.payload, r.hit);
}

// The 16-byte vrt_hit record as one vector store.  kGlsl: t is the biased tmin and
// the face the first axis with tmin >= side (hit.normal's sideMask, VoxelTraversal.glsl:190).
template <bool kGlsl = false>
__device__ __forceinline__ uint4 pack_hit(const TraceResult& r, float dx, float dy, float dz, uint32_t tag) {
    if (!r.hit) return make_uint4(VRT_MISS_VOXEL, VRT_MISS_FACE | (r.steps << 16), 0x7F800000u, tag);
    float t;
    uint32_t face;
    if (kGlsl) {
        t = r.tb;
        if (t >= r.sx)
            face = dx < 0.0f ? 1u : 0u;
        else if (t >= r.sy)
            face = dy < 0.0f ? 3u : 2u;
        else
            face = dz < 0.0f ? 5u : 4u;
    } else {
        t = min_x86(min_x86(r.sx, r.sy), r.sz);
        if (r.sx == t)
            face = dx < 0.0f ? 1u : 0u;
        else if (r.sy == t)
            face = dy < 0.0f ? 3u : 2u;
        else
            face = dz < 0.0f ? 5u : 4u;
    }
    return make_uint4(r.voxel, face | r.material << 8 | r.steps << 16, __float_as_uint(t), tag);
}

__device__ __forceinline__ uint4 no_ray_hit() {
    return make_uint4(VRT_MISS_VOXEL, VRT_MISS_FACE, 0x7F800000u, VRT_NO_RAY);
}

// HitResult.Normal (CpuRenderer.cpp:213-217) and origin = Pos + Normal*0.01 (:389).
// kGlsl: hit.normal = mix(0, -sign(dir), tmin >= sideDist) (VoxelTraversal.glsl:190-192),
// every axis within the bias, sign(+-0) = 0.
template <bool kGlsl = false>
__device__ __forceinline__ void secondary_origin(const TraceResult& r, float dx, float dy, float dz, float& ox,
                                                 float& oy, float& oz, float& nx, float& ny, float& nz) {
    if (kGlsl) {
        nx = r.tb >= r.sx ? (dx > 0.0f ? -1.0f : (dx < 0.0f ? 1.0f : 0.0f)) : 0.0f;
        ny = r.tb >= r.sy ? (dy > 0.0f ? -1.0f : (dy < 0.0f ? 1.0f : 0.0f)) : 0.0f;
        nz = r.tb >= r.sz ? (dz > 0.0f ? -1.0f : (dz < 0.0f ? 1.0f : 0.0f)) : 0.0f;
    } else {
        const float t = min_x86(min_x86(r.sx, r.sy), r.sz);
        const bool mx = r.sx == t, my = r.sy == t, mz = !mx && !my;
        nx = mx ? (signbit(dx) ? 1.0f : -1.0f) : 0.0f;
        ny = my ? (signbit(dy) ? 1.0f : -1.0f) : 0.0f;
        nz = mz ? (signbit(dz) ? 1.0f : -1.0f) : 0.0f;
    }
    ox = __fadd_rn(r.cx, __fmul_rn(nx, 0.01f));
    oy = __fadd_rn(r.cy, __fmul_rn(ny, 0.01f));
    oz = __fadd_rn(r.cz, __fmul_rn(nz, 0.01f));
}

}  // namespace vrt

namespace vrt {

// PCG32 (O'Neill, pcg-random.org: 64-bit LCG state, XSH-RR output).
struct DevPcg32 {
    uint64_t state, inc;
    __device__ __forceinline__ DevPcg32(uint64_t initstate, uint64_t initseq) {
        state = 0;
        inc = (initseq << 1) | 1u;
        next();
        state += initstate;
        next();
    }
    __device__ __forceinline__ uint32_t next() {
        const uint64_t old = state;
        state = old * 6364136223846793005ULL + inc;
        const uint32_t xs = (uint32_t)(((old >> 18) ^ old) >> 27);
        const uint32_t rot = (uint32_t)(old >> 59);
        return (xs >> rot) | (xs << ((32 - rot) & 31));
    }
    // uniform in [-1, 1) with 2^-23 spacing; every op exact
    __device__ __forceinline__ float next_signed() {
        return __fsub_rn(__fmul_rn(__uint2float_rn(next() >> 8), 0x1p-23f), 1.0f);
    }
};

constexpr uint64_t kBounceStream = 0x9E3779B97F4A7C15ULL;

// Lambertian bounce normalize(n + s), s uniform on the sphere by rejection from the
// cube (the structure of CpuRenderer.cpp:392 with IEEE-exact sampling).  At most 64 samples in
// all.  The rejection is a loop of its own: half the samples are taken, so the lanes of a warp
// leave it at 5 to 6 different iterations, and with the square roots and divisions inside they
// ran once for each (two 720p views of 4 bounces 404 -> 372 us, an anisotropic path batch
// 694 -> 654).
__device__ __forceinline__ void bounce_dir(uint32_t pixel, uint32_t bounce, float nx, float ny, float nz, float& dx,
                                           float& dy, float& dz) {
    DevPcg32 rng(pixel ^ bounce, kBounceStream);
    for (int left = 64; left > 0;) {
        float x, y, z, r2;
        bool in;
        do {
            x = rng.next_signed();
            y = rng.next_signed();
            z = rng.next_signed();
            r2 = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
            in = r2 > 1e-6f && r2 <= 1.0f;
        } while (--left > 0 && !in);
        if (!in) break;
        const float r = __fsqrt_rn(r2);
        const float ax = __fadd_rn(nx, __fdiv_rn(x, r)), ay = __fadd_rn(ny, __fdiv_rn(y, r)),
                    az = __fadd_rn(nz, __fdiv_rn(z, r));
        const float l2 = __fadd_rn(__fadd_rn(__fmul_rn(ax, ax), __fmul_rn(ay, ay)), __fmul_rn(az, az));
        if (!(l2 > 1e-12f)) continue;
        const float l = __fsqrt_rn(l2);
        dx = __fdiv_rn(ax, l);
        dy = __fdiv_rn(ay, l);
        dz = __fdiv_rn(az, l);
        return;
    }
    const float l = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz)));
    dx = __fdiv_rn(nx, l);
    dy = __fdiv_rn(ny, l);
    dz = __fdiv_rn(nz, l);
}

// Hit record from a finished RayState (steps = iteration index at exit).
template <bool kGlsl = false>
__device__ __forceinline__ uint4 pack_state(const RayState& s, uint32_t material, bool hit, uint32_t steps,
                                           uint32_t tag) {
    TraceResult r;
    r.sx = s.sx;
    r.sy = s.sy;
    r.sz = s.sz;
    r.tb = s.tb;
    r.voxel = s.hit_voxel();
    r.steps = steps;
    r.material = material;
    r.hit = hit;
    return pack_hit<kGlsl>(r, s.dx, s.dy, s.dz, tag);
}

// Where the secondary rays of a hit start and the hit's normal (secondary_origin).
template <bool kGlsl = false>
__device__ __forceinline__ void hit_frame(const RayState& s, float& ox, float& oy, float& oz, float& nx, float& ny,
                                          float& nz) {
    TraceResult r;
    r.cx = s.cx;
    r.cy = s.cy;
    r.cz = s.cz;
    r.sx = s.sx;
    r.sy = s.sy;
    r.sz = s.sz;
    r.tb = s.tb;
    secondary_origin<kGlsl>(r, s.dx, s.dy, s.dz, ox, oy, oz, nx, ny, nz);
}

// The GPU renderer's whole path (VoxelRender.comp:51-86), a view with a sun direction
// and bounces: record plane k >= 1 holds a sun ray for k = 1, 3, 5 (after the primary
// hit and the first two bounce hits) and otherwise bounce k/2 (k <= 4) or k - 3
// (k >= 6).  Flag in ViewDev::path.
constexpr uint32_t kPathFull = 1u << 20;
__host__ __device__ __forceinline__ bool full_is_sun(uint32_t k) { return k <= 5u && (k & 1u); }
__host__ __device__ __forceinline__ uint32_t full_bounce(uint32_t k) { return k <= 4u ? k >> 1 : k - 3u; }

// Origin and direction of the next ray of a path after a hit: the shadow ray
// (kind 1 with shadows) or bounce `bounce` (1-based).
template <bool kGlsl = false>
__device__ __forceinline__ void next_path_ray(const RayState& s, bool shadow, const float* sun, uint32_t pixel,
                                              uint32_t bounce, float& ox, float& oy, float& oz, float& dx, float& dy,
                                              float& dz) {
    TraceResult r;
    r.cx = s.cx;
    r.cy = s.cy;
    r.cz = s.cz;
    r.sx = s.sx;
    r.sy = s.sy;
    r.sz = s.sz;
    r.tb = s.tb;
    float nx, ny, nz;
    secondary_origin<kGlsl>(r, s.dx, s.dy, s.dz, ox, oy, oz, nx, ny, nz);
    if (shadow) {
        dx = sun[0];
        dy = sun[1];
        dz = sun[2];
    } else {
        bounce_dir(pixel, bounce, nx, ny, nz, dx, dy, dz);
    }
}

}  // namespace vrt

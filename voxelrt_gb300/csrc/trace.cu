// trace.cu - per-view and explicit-ray traversal kernels and their C ABI.
//
// vrt_render_view* is the one-launch-per-view path of GpuRenderer::RenderFrame
// (src/VoxelRT/GpuRenderer.cpp:239-273): thread blocks over 16x8 pixels of the image, fewer
// of a small one (thin_launch.cuh), one primary ray per pixel (Shaders/VoxelRender.comp:27-30),
// writing a headless hit buffer instead of the G-buffer.  vrt_cast* traverses caller-supplied rays.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "cast_queue.h"
#include "thin_launch.cuh"
#include "trace_core.cuh"
#include "world.h"

namespace vrt {
namespace {

uint32_t eff_iters(uint32_t max_iters, bool glsl = false) {
    if (max_iters == 0) return glsl ? VRT_GLSL_MAX_ITERS : VRT_DEFAULT_MAX_ITERS;
    return max_iters > 65535u ? 65535u : max_iters;
}

// One thread per pixel (thin_pixel).  Bound by the latency of its steps: with leave for 48 registers
// (the compiler's choice is 32) frames of a terrain take 3 to 8 % less (64x64 of a 256-voxel one
// 14.3 -> 13.8 us, 192x192 15.3 -> 14.0, 512x512 16.1 -> 15.5).
// inside: the camera origin is (origin_inside_near)
__global__ void __maxnreg__(48) render_view_kernel(const __grid_constant__ DevWorld w,
                                                        const __grid_constant__ vrt_camera cam,
                                                        const __grid_constant__ ClipBox clip, bool inside,
                                                        uint32_t lanes_log2, uint32_t max_iters,
                                                        uint4* __restrict__ out) {
    uint32_t px, py;
    if (!thin_pixel<true>(lanes_log2, px, py) || px >= cam.width || py >= cam.height) return;
    float dx, dy, dz;
    camera_ray(cam, px, py, dx, dy, dz);
    const int32_t wox = cam.world_origin[0], woy = cam.world_origin[1], woz = cam.world_origin[2];
    RayState s;
    if (inside)
        ray_start_inside<false>(s, cam.origin[0], cam.origin[1], cam.origin[2], dx, dy, dz, wox, woy, woz);
    else
        ray_start<false>(s, clip, cam.origin[0], cam.origin[1], cam.origin[2], dx, dy, dz, wox, woy, woz);
    TraceCounters cnt;
    uint32_t i = 0;
    const bool hit =
        dda_steps_mode<false, false>(s, w, wox, woy, woz, cnt, false, false, false, 0, i, max_iters) == kStepHit;
    const uint32_t pix = py * cam.width + px;
    out[pix] = pack_state<false>(s, hit_material(s, w.payload, hit), hit, i, pix);
}

// A thread per ray, stalled rays looked for every `slice` steps: 16, and 8 for GLSL rays.  For
// rayCastCoarse's, which are looked at from iteration 31 on alone, 131,072 random rays in a mixed world
// with 8 / 16 / 32 steps 14.6 / 14.2 / 14.1 us (14.0 without the test), 120,000 with anisotropic LODs in a
// world with 2 % of its voxels set 35.3 / 35.3 / 41.5 us (45.6 without).
template <bool kGlsl, bool kAniso = false>
__global__ void __launch_bounds__(256) cast_kernel(const __grid_constant__ DevWorld w,
                                                  const __grid_constant__ ClipBox clip,
                                                  const float4* __restrict__ rays, uint32_t n, int32_t wox,
                                                  int32_t woy, int32_t woz, uint32_t max_iters,
                                                  uint4* __restrict__ out, bool coarse, uint32_t lanes_log2,
                                                  uint32_t slice) {
    if constexpr (kAniso) fill_forward_lut();
    const uint32_t lane = threadIdx.x & 31;
    if (lane >> lanes_log2) return;
    const uint32_t i = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5 << lanes_log2) + lane;
    if (i >= n) return;
    const float4 a = rays[2 * (size_t)i], b = rays[2 * (size_t)i + 1];
    RayState s;
    ray_start<kGlsl>(s, clip, a.x, a.y, a.z, a.w, b.x, b.y, wox, woy, woz, coarse);
    uint32_t k = 0;
    const bool hit =
        dda_trace<kGlsl, !kGlsl>(s, w, wox, woy, woz, coarse, coarse, kAniso, k, max_iters, slice) == kStepHit;
    out[i] = pack_state<kGlsl>(s, hit_material(s, w.payload, hit), hit, k, __float_as_uint(b.z));
}

// Explicit rays whose lengths vary widely (random origins and directions: some hit at
// once, others run to the iteration cap) leave most lanes of a thread-per-ray warp idle
// behind its longest ray.  Here each warp walks its own grid-strided sequence of 32-ray
// chunks (warp g takes rays [32 (g + k G), +32) for k = 0, 1, ...), traces in slices
// of `inner` DDA steps, and once fewer than `refill` lanes trace stores the records of the
// rays that ended and refills those lanes from its chunks.  No
// device queue: calls on different streams stay independent.  Same records as
// cast_kernel: a lane's steps continue from where its ray left off, and a ray's record
// is packed from the state at its exit.
template <bool kGlsl, bool kAniso = false>
__global__ void __maxnreg__(56) cast_persistent_kernel(const __grid_constant__ DevWorld w,
                                                             const __grid_constant__ ClipBox clip,
                                                             const float4* __restrict__ rays, uint32_t n,
                                                             int32_t wox, int32_t woy, int32_t woz, uint32_t max_iters,
                                                             uint32_t inner, uint32_t refill, uint4* __restrict__ out,
                                                             bool coarse) {
    if constexpr (kAniso) fill_forward_lut();
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    const uint32_t stride = (gridDim.x * blockDim.x) & ~31u;  // rays between a warp's chunks
    uint32_t next = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;  // first ray of the warp's next chunk
    uint32_t q_next = 0, q_end = 0;
    bool active = false, ended = false, hit = false;
    uint32_t ri = 0, iter = 0, tag = 0;
    float t0 = 0.0f;
    RayState s;
    TraceCounters cnt{0, 0};
    for (;;) {
        // The material of a ray that ended and the ray that takes its lane are loaded together,
        // before the record is stored: one wait for memory a round in place of two.
        uint32_t material = 0, rn = 0;
        if (ended) {
            material = hit_material(s, w.payload, hit);
            active = false;
        }
        const uint32_t act = __ballot_sync(0xffffffffu, active);
        bool mine = false;
        if ((uint32_t)__popc(act) < refill) {
            uint32_t idle = ~act;
            while (idle) {
                if (q_next >= q_end) {
                    if (next >= n) break;
                    q_next = next;
                    q_end = chunk_end(next, n);
                    next = chunk_after(next, stride, n);
                }
                const uint32_t take = min(q_end - q_next, (uint32_t)__popc(idle));
                const uint32_t rank = __popc(idle & lt);
                const bool now = ((idle >> lane) & 1u) && rank < take;
                if (now) {
                    rn = q_next + rank;
                    mine = true;
                }
                idle &= ~__ballot_sync(0xffffffffu, now);
                q_next += take;
            }
        }
        float4 a{}, b{};
        if (mine) {
            a = __ldg(rays + 2 * (size_t)rn);
            b = __ldg(rays + 2 * (size_t)rn + 1);
        }
        if (ended) {
            out[ri] = pack_state<kGlsl>(s, material, hit, iter, tag);
            ended = false;
        }
        if (mine) {
            ri = rn;
            tag = __float_as_uint(b.z);
            ray_start<kGlsl>(s, clip, a.x, a.y, a.z, a.w, b.x, b.y, wox, woy, woz, coarse);
            iter = 0;
            t0 = no_t();
            active = true;
        }
        if (__ballot_sync(0xffffffffu, active) == 0) break;
        // slices until fewer than `refill` lanes are tracing
        do {
            if (active && !ended) {
                const uint32_t first = iter, lim = max_iters - iter < inner ? max_iters : iter + inner;
                // GLSL variants (rayCastCoarse, anisotropic LODs) are uniform over the launch
                const uint32_t st = dda_steps_mode<false, kGlsl, true>(s, w, wox, woy, woz, cnt, coarse, coarse, kAniso,
                                                                       0, iter, lim);
                if (st == kStepContinue && stalled<kGlsl>(s, t0, coarse, first)) iter = max_iters;
                t0 = last_t<kGlsl>(s);
                if (st != kStepContinue || iter >= max_iters) {
                    ended = true;
                    hit = st == kStepHit;
                }
            }
        } while ((uint32_t)__popc(__ballot_sync(0xffffffffu, active && !ended)) >= refill);
    }
}

vrt_status check_camera(const vrt_camera* cam) {
    if (!cam || cam->width == 0 || cam->height == 0 || cam->width > 16384 || cam->height > 16384 ||
        !world_origin_ok(cam->world_origin)) {
        set_error("camera must be 1..16384 pixels on each side with |world origin| <= 2^30");
        return VRT_ERR_INVALID_ARG;
    }
    return VRT_OK;
}

vrt_status launch_render(vrt_world* w, const vrt_camera* cam, uint32_t max_iters, vrt_hit* hits,
                         cudaStream_t stream) {
    const uint32_t ll = thin_lanes_log2((uint64_t)cam->width * cam->height, sm_count());
    L2Window l2;
    vrt_status st = l2.enter(w, stream);
    if (st != VRT_OK) return st;
    const DevWorld dw = w->dev();
    const float* o = cam->origin;
    const ClipBox clip = clip_box(dw, cam->world_origin);
    render_view_kernel<<<thin_grid(ll, cam->width, cam->height), kFrameThreads, 0, stream>>>(
        dw, *cam, clip, origin_inside_near(clip, o[0], o[1], o[2]), ll, eff_iters(max_iters),
        reinterpret_cast<uint4*>(hits));
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

// Launch shape of cast_persistent_kernel.  A slice's end costs about as much as a step, and lanes
// whose rays have ended, or stand still (stalled), wait for it: short slices where rays end early or
// stand still, longer ones where they are long and no slice finds a stalled ray.  On 4.2 M random
// rays, launches repeated on the same rays:
// - CPU traversal, slices of 4 / 5 / 6 / 8: 512-voxel mixed world 238 / 241 / 243 / 251 us, terrain
//   232 / 225 / 222 / 224, a world with 2 % of its voxels set 462 / 445 / 432 / 413 (1 M of them 150 /
//   144 / 140 / 134, as 147 with slices of 12 and no test for stalled rays);
// - GLSL, 4 / 6 / 8: 208 / 227 / 250, 198 / 211 / 227, 280 / 296 / 322 us; anisotropic LODs alike;
// - rayCastCoarse, whose rays are looked at from iteration 31 on alone, 4 / 8 / 12: 255 / 270 /
//   284, 242 / 246 / 271, 602 / 532 / 527; with anisotropic LODs, 4 / 5 / 8: 192 / 196 / 221,
//   257 / 259 / 284, 497 / 480 / 453 (504 us before the slices went on until a refill).
constexpr uint32_t kCastThreads = 128, kCastRefill = 28;
constexpr uint32_t cast_slice(bool glsl, bool coarse, bool aniso) {
    return coarse ? (aniso ? 5u : 8u) : glsl ? 4u : 5u;
}
// Below this many rays the thread-per-ray kernel is used: too few rays to fill the persistent
// grid's lanes several times.  400,000 random CPU rays 36 us against 40 (terrain) and 20 against
// 24 (mixed world), 800,000 rays 60 and 34 against 57 and 35, and twice as fast on coherent ones at
// any count; 400,000 anisotropic rays 42 and 34 us against 40 and 27.
constexpr uint32_t kCastPersistentMin = 3u << 18, kCastPersistentMinGlsl = 1u << 18;

vrt_status launch_cast(vrt_world* w, const vrt_ray* rays, uint32_t n, const vrt_cast_params* p, vrt_hit* hits,
                       cudaStream_t stream) {
    if (n == 0) return VRT_OK;
    const bool glsl = (p->flags & VRT_CAST_GLSL) != 0, coarse = (p->flags & VRT_CAST_GLSL_COARSE) != 0,
               aniso = (p->flags & VRT_CAST_GLSL_ANISO) != 0;
    const float4* r4 = reinterpret_cast<const float4*>(rays);
    uint4* o4 = reinterpret_cast<uint4*>(hits);
    uint32_t iters = eff_iters(p->max_iters, glsl);
    if (coarse) iters = std::min<uint32_t>(iters, VRT_GLSL_COARSE_MAX_ITERS);
    const DevWorld dw = w->dev();
    const ClipBox clip = clip_box(dw, p->world_origin);
    L2Window l2;
    vrt_status st = l2.enter(w, stream);
    if (st != VRT_OK) return st;
    if (n < (glsl ? kCastPersistentMinGlsl : kCastPersistentMin)) {
        auto kernel = glsl ? (aniso ? cast_kernel<true, true> : cast_kernel<true>) : cast_kernel<false>;
        const uint32_t ll = thin_lanes_log2(n, sm_count()), per_block = 8u << ll;
        kernel<<<(n + per_block - 1) / per_block, 256, 0, stream>>>(dw, clip, r4, n, p->world_origin[0],
                                                                    p->world_origin[1], p->world_origin[2], iters, o4,
                                                                    coarse, ll, glsl && !coarse ? 8 : 16);
    } else {
        auto kernel = glsl ? (aniso ? cast_persistent_kernel<true, true> : cast_persistent_kernel<true>)
                           : cast_persistent_kernel<false>;
        int dev = 0, sms = 0, occ = 0;
        VRT_CUDA(cudaGetDevice(&dev));
        VRT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        VRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kCastThreads, 0));
        const uint32_t blocks = (uint32_t)(sms * std::max(occ, 1));
        kernel<<<blocks, kCastThreads, 0, stream>>>(dw, clip, r4, n, p->world_origin[0], p->world_origin[1],
                                                    p->world_origin[2], iters, cast_slice(glsl, coarse, aniso),
                                                    kCastRefill, o4, coarse);
    }
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

vrt_status check_params(const vrt_cast_params* p) {
    const uint32_t glsl_opts = VRT_CAST_GLSL_COARSE | VRT_CAST_GLSL_ANISO;
    if (!p || (p->flags & ~(VRT_CAST_GLSL | glsl_opts)) != 0 ||
        ((p->flags & glsl_opts) && !(p->flags & VRT_CAST_GLSL)) || !world_origin_ok(p->world_origin)) {
        set_error("cast params missing, flags other than VRT_CAST_GLSL [| VRT_CAST_GLSL_COARSE | "
                  "VRT_CAST_GLSL_ANISO], or |world origin| > 2^30");
        return VRT_ERR_INVALID_ARG;
    }
    return VRT_OK;
}

}  // namespace
}  // namespace vrt

using namespace vrt;

extern "C" {

vrt_status vrt_cast_device(vrt_world* w, const vrt_ray* rays, uint32_t n, const vrt_cast_params* params,
                           vrt_hit* hits, void* stream) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK || (st = check_params(params)) != VRT_OK) return st;
    if (n && (!rays || !hits)) {
        set_error("null ray or hit buffer");
        return VRT_ERR_INVALID_ARG;
    }
    return launch_cast(w, rays, n, params, hits, (cudaStream_t)stream);
}

vrt_status vrt_cast(vrt_world* w, const vrt_ray* rays, uint32_t n, const vrt_cast_params* params, vrt_hit* hits,
                    void* stream_) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK || (st = check_params(params)) != VRT_OK) return st;
    if (n == 0) return VRT_OK;
    if (!rays || !hits) {
        set_error("null ray or hit buffer");
        return VRT_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(w->mu);
    cudaStream_t stream = (cudaStream_t)stream_;
    const size_t rb = (size_t)n * sizeof(vrt_ray), hb = (size_t)n * sizeof(vrt_hit);
    VRT_CUDA(w->d_io.reserve(rb + hb));
    vrt_ray* d_rays = (vrt_ray*)w->d_io.ptr;
    vrt_hit* d_hits = (vrt_hit*)((uint8_t*)w->d_io.ptr + rb);
    VRT_CUDA(cudaMemcpyAsync(d_rays, rays, rb, cudaMemcpyHostToDevice, stream));
    if ((st = launch_cast(w, d_rays, n, params, d_hits, stream)) != VRT_OK) return st;
    VRT_CUDA(cudaMemcpyAsync(hits, d_hits, hb, cudaMemcpyDeviceToHost, stream));
    VRT_CUDA(cudaStreamSynchronize(stream));
    return VRT_OK;
}

vrt_status vrt_render_view_device(vrt_world* w, const vrt_camera* cam, uint32_t max_iters, vrt_hit* hits,
                                  void* stream) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK || (st = check_camera(cam)) != VRT_OK) return st;
    if (!hits) {
        set_error("null hit buffer");
        return VRT_ERR_INVALID_ARG;
    }
    return launch_render(w, cam, max_iters, hits, (cudaStream_t)stream);
}

vrt_status vrt_render_view(vrt_world* w, const vrt_camera* cam, uint32_t max_iters, vrt_hit* hits, void* stream_) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK || (st = check_camera(cam)) != VRT_OK) return st;
    if (!hits) {
        set_error("null hit buffer");
        return VRT_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(w->mu);
    cudaStream_t stream = (cudaStream_t)stream_;
    const size_t hb = (size_t)cam->width * cam->height * sizeof(vrt_hit);
    VRT_CUDA(w->d_io.reserve(hb));
    if ((st = launch_render(w, cam, max_iters, (vrt_hit*)w->d_io.ptr, stream)) != VRT_OK) return st;
    VRT_CUDA(cudaMemcpyAsync(hits, w->d_io.ptr, hb, cudaMemcpyDeviceToHost, stream));
    VRT_CUDA(cudaStreamSynchronize(stream));
    return VRT_OK;
}

}  // extern "C"

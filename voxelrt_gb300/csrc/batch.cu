// batch.cu - view paths (primary + shadow / diffuse bounces) and the batched
// persistent traversal over many worlds and views.
//
// The reference dispatches one VoxelRender.comp per frame (GpuRenderer.cpp:267-268)
// with one invocation per pixel tracing its whole path (VoxelRender.comp:27-93).
// vrt_render_path keeps that structure (the per-view baseline).  vrt_batch_* puts
// the views of many worlds behind one device queue of ray tiles that persistent warps
// take.  Without bounces (tile_kernel) a warp traces 32 pixels of a tile to their ends; with
// bounces (persistent_kernel) it hands rays to idle lanes (regeneration), refills when fewer
// than `refill_threshold` lanes are still tracing (compaction), and a lane that finishes a ray
// continues its pixel's path in place.

#include <cuda_runtime.h>

#include <cuda/atomic>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "batch_internal.h"
#include "thin_launch.cuh"
#include "trace_core.cuh"
#include "world.h"

namespace vrt {
namespace {

__device__ __forceinline__ uint32_t compact_even_bits(uint32_t k) {
    k &= 0x55u;
    k = (k | (k >> 1)) & 0x33u;
    k = (k | (k >> 2)) & 0x0Fu;
    return k;
}

// What the rays of one view share, from its camera origin: whether that is inside and near
// (origin_inside_near), and (tile_kernel, CPU traversal) what iteration 0 finds there: the
// origin's voxel in biased form and the alignment mask of its cell, or that it is solid.
constexpr uint32_t kStartUnknown = 0xFFFFFFFFu, kStartSolid = 0xFFFFFFFEu;
struct ViewStart {
    ClipBox clip;
    uint32_t inside;
    uint32_t mask;      // kStartUnknown, kStartSolid or the alignment mask
    uint32_t voxel[3];
    uint32_t material;  // of a solid origin
};

VRT_HD inline ViewStart view_start(const DevWorld& w, const ViewDev& v) {
    ViewStart s{};
    s.clip = clip_box(w, v.wo);
    s.inside = origin_inside_near(s.clip, v.ox, v.oy, v.oz) ? 1u : 0u;
    s.mask = kStartUnknown;
    return s;
}

// Store of record i: the 16-byte record, or with kPacked its 12-byte form (vrt_hit_packed).
template <bool kPacked>
__device__ __forceinline__ void store_record(uint4* __restrict__ out, uint64_t i, uint4 r) {
    if constexpr (kPacked) {
        uint32_t* o = reinterpret_cast<uint32_t*>(out) + 3 * i;
        o[0] = r.x;
        o[1] = r.w == VRT_NO_RAY ? (r.y & 0xFFFF00FFu) | (VRT_PACKED_NO_RAY << 8) : r.y;
        o[2] = r.z;
    } else {
        out[i] = r;
    }
}

// One pixel's whole path: the primary ray, then its sun ray or bounces, or with kFull the GPU
// renderer's path (VoxelRender.comp:27-93); returns the rays traced.  One loop over the rays,
// so that the step loop is compiled once.
template <bool kGlsl, bool kAniso, bool kBounces, bool kPacked, bool kFar = false>
__device__ __forceinline__ uint32_t trace_pixel(const ViewDev& v, const DevWorld& w, const ViewStart& vs, uint32_t px,
                                                uint32_t py, uint4* __restrict__ out) {
    const uint32_t pixel = py * v.width + px, last = v.last_kind();
    uint64_t o = v.out_base + pixel;
    float dx, dy, dz;
    camera_ray(v.d0, v.du, v.dv, px, py, dx, dy, dz);
    if (!kGlsl && !kBounces && vs.mask == kStartSolid && last == 0) {
        // the camera stands in a solid voxel: every ray hits it on iteration 0 at t = 0, face X
        const uint32_t x = vs.voxel[0] - kVoxelBias, y = vs.voxel[1] - kVoxelBias, z = vs.voxel[2] - kVoxelBias;
        store_record<kPacked>(
            out, o, make_uint4(x | y << 11 | z << 21, (dx < 0.0f ? 1u : 0u) | vs.material << 8, 0u, pixel));
        return 1;
    }
    const int32_t wox = v.wo[0], woy = v.wo[1], woz = v.wo[2];
    const bool full = kBounces && (v.path & kPathFull) != 0;
    RayState s;
    uint32_t i = 0;
    if (vs.inside) {
        ray_start_inside<kGlsl>(s, v.ox, v.oy, v.oz, dx, dy, dz, wox, woy, woz);
        if (!kGlsl && !kBounces && vs.mask < kStartSolid && s.fast) {
            step_on<true, false, false>(s, vs.voxel[0], vs.voxel[1], vs.voxel[2], vs.mask, wox, woy, woz, 0);
            i = 1;
        }
    } else {
        ray_start<kGlsl>(s, vs.clip, v.ox, v.oy, v.oz, dx, dy, dz, wox, woy, woz);
    }
    TraceCounters cnt{0, 0};
    float hx = 0.0f, hy = 0.0f, hz = 0.0f, nx = 0.0f, ny = 0.0f, nz = 0.0f;  // the last hit frame
    for (uint32_t k = 0;;) {
        // GLSL mode: shadow and bounce rays are rayCastCoarse's (VoxelRender.comp:56,74)
        const bool coarse = kGlsl && k != 0;
        const uint32_t iters = coarse ? min(v.max_iters, kCoarseMaxIters) : v.max_iters;
        uint32_t st;
        if constexpr (kFar)
            st = dda_trace<kGlsl, false>(s, w, wox, woy, woz, coarse, coarse, kAniso, i, iters, 16);
        else
            st = dda_steps_mode<false, kGlsl>(s, w, wox, woy, woz, cnt, coarse, coarse, kAniso, 0, i, iters);
        const bool hit = st == kStepHit;
        store_record<kPacked>(out, o, pack_state<kGlsl>(s, hit_material(s, w.payload, hit), hit, i, pixel));
        if (k == last) return k + 1;
        // the path goes on after a hit, and the whole path after a sun ray, hit or miss
        const bool go = hit || (full && full_is_sun(k));
        const size_t plane = (size_t)v.width * v.height;
        if (!go) {
            const uint32_t n = k + 1;
            for (; k < last; k++) store_record<kPacked>(out, o += plane, no_ray_hit());
            return n;
        }
        k++;
        o += plane;
        if (kBounces) {
            // a sun ray starts from the hit just traced; a bounce from the hit before its
            // sun ray (kept), or from the bounce just traced when no sun ray follows it
            if (!full || full_is_sun(k) || !full_is_sun(k - 1)) hit_frame<kGlsl>(s, hx, hy, hz, nx, ny, nz);
            if (full ? full_is_sun(k) : v.shadow() != 0) {
                dx = v.sun[0];
                dy = v.sun[1];
                dz = v.sun[2];
            } else {
                bounce_dir(pixel, full ? full_bounce(k) : k, nx, ny, nz, dx, dy, dz);
            }
        } else {
            hit_frame<kGlsl>(s, hx, hy, hz, nx, ny, nz);
            dx = v.sun[0];
            dy = v.sun[1];
            dz = v.sun[2];
        }
        ray_start<kGlsl>(s, vs.clip, hx, hy, hz, dx, dy, dz, wox, woy, woz, kGlsl);
        i = 0;
    }
}

// One thread per pixel (thin_pixel), whole path (VoxelRender.comp:27-93 structure).  kBounces: the
// view has bounces; without them 48 registers in place of 56 (a 1080p frame with its sun
// ray: 121.6 -> 118.0 us).  kFar: the world origin is not near; most rays stand still, and dda_trace
// ends them (720p with sun rays from 2^22 voxels off, GLSL: 592 -> 148 us, CPU traversal 322 -> 113).
template <bool kGlsl, bool kAniso, bool kBounces, bool kThin, bool kFar>
__global__ void __launch_bounds__(kFrameThreads)
    view_path_kernel(const __grid_constant__ DevWorld w, const __grid_constant__ ViewDev v,
                     const __grid_constant__ ViewStart vs, uint32_t lanes_log2, uint4* __restrict__ out) {
    if constexpr (kAniso) fill_forward_lut();
    uint32_t px, py;
    if (!thin_pixel<kThin>(lanes_log2, px, py) || px >= v.width || py >= v.height) return;
    trace_pixel<kGlsl, kAniso, kBounces, false, kFar>(v, w, vs, px, py, out);
}

// View-table loads: read-only through the non-coherent path, or at L2 (coherent with
// the host's copies) for a resident launch, whose table grows while it runs.
template <bool kResident, typename T>
__device__ __forceinline__ T ldv(const T* p) {
    if (kResident) return __ldcg(p);
    return __ldg(p);
}

// A view-table field: from the warp's shared copy (`shared`, resident launches only),
// else from global memory.
template <bool kResident, typename T>
__device__ __forceinline__ T vget(const T* a, bool shared) {
    if (!kResident) return __ldg(a);
    return shared ? *a : __ldcg(a);
}

// A 16-byte (or 8-byte) group of view-table fields: from global memory through the
// read-only path, or from the warp's shared copy (resident launches).
template <bool kResident, typename V>
__device__ __forceinline__ V vget4(const V* a) {
    if (!kResident) return __ldg(a);
    return *a;
}

// A world-table entry (the table does not change while a launch runs).
__device__ __forceinline__ DevWorld load_world(const DevWorld* p) {
    DevWorld w;
    const uint4* a = reinterpret_cast<const uint4*>(p);
    uint4* b = reinterpret_cast<uint4*>(&w);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(DevWorld) / 16); i++) b[i] = __ldg(a + i);
    return w;
}

constexpr uint32_t kClaimEmpty = 0xFFFFFFFFu, kClaimStop = 0xFFFFFFFEu;

constexpr uint32_t kNoChunk = 0xFFFFFFFFu;

// Resident launch: per-warp state of the mailbox protocol, kept in shared memory and
// used by lane 0 alone (warp-uniform values in registers would cost every lane a
// register in the traversal loop).
struct ResidentWarp {
    uint32_t pub_chunks, pub_views;  // last hint word read
    uint32_t pend;                   // reserved chunk number not yet published, or kNoChunk
    uint32_t backoff;                // rounds until an empty mailbox is re-read
    uint32_t idle_ns, sleep_ns;      // sleep while idle
    uint32_t acc_view, acc_n;        // finished pixels of view acc_view not yet subtracted
    uint32_t cached_view;            // view held in the warp's shared copy of the table entry
    uint32_t q_inside;               // origin_inside_near() for that view's camera
};
constexpr uint32_t kNoView = 0xFFFFFFFFu;

// Resident launch, lane 0: the next chunk to trace.  Chunk numbers come from one
// atomicAdd (no retries under contention); a number the host has not published yet
// stays reserved in `pend` until it is (kClaimEmpty meanwhile), or until the mailbox
// is closed below it (kClaimStop: a closed word's chunk count is final, nothing is
// published after a close).  Published counts come from the device copy of the
// mailbox word (the hint): it is never ahead of the mailbox, and the host writes it
// only after the views it counts are uploaded, so the warps never read host memory
// to claim (thousands of them reading one host word at once would queue on the host
// link).  While the warp still has lanes tracing (`busy`), an empty mailbox is
// re-read only every 8 rounds.
__device__ __forceinline__ uint32_t resident_claim(const BatchParams& p, ResidentWarp& rw, bool busy) {
    if (busy && rw.backoff > 0) {
        rw.backoff--;
        return kClaimEmpty;
    }
    const uint32_t n = rw.pend != kNoChunk ? rw.pend : atomicAdd(p.next_chunk, 1u);
    if (n >= rw.pub_chunks) {
        const unsigned long long h =
            cuda::atomic_ref<const unsigned long long, cuda::thread_scope_device>(*p.hint).load(
                cuda::memory_order_acquire);
        rw.pub_chunks = (uint32_t)h;
        rw.pub_views = (uint32_t)(h >> 32) & 0x7FFFFFFFu;
        if (n >= rw.pub_chunks) {
            if (h & kMailboxClosed) {
                rw.pend = kNoChunk;
                return kClaimStop;
            }
            rw.pend = n;
            rw.backoff = 8;
            return kClaimEmpty;
        }
    }
    rw.pend = kNoChunk;
    return n;
}

// Resident launch, lane 0 of an idle warp that has claimed every chunk it saw
// published: close the mailbox unless more work was published since the hint word
// in pub_chunks / pub_views.  True when the mailbox is closed with nothing left to
// claim.  On a failed close nothing is adopted from the mailbox word: it can count
// views whose uploads are still in flight, so published counts come from the hint
// alone (the next claim re-reads it).
__device__ __forceinline__ bool resident_try_close(const BatchParams& p, uint32_t pub_chunks, uint32_t pub_views) {
    const unsigned long long seen = mailbox_word(pub_chunks, pub_views);
    unsigned long long expected = seen;
    cuda::atomic_ref<unsigned long long, cuda::thread_scope_system> mb(*p.mailbox);
    if (mb.compare_exchange_strong(expected, seen | kMailboxClosed, cuda::memory_order_acq_rel)) {
        // the other warps learn of the close from the hint (same value the host would write)
        cuda::atomic_ref<unsigned long long, cuda::thread_scope_device>(*const_cast<unsigned long long*>(p.hint))
            .store(seen | kMailboxClosed, cuda::memory_order_relaxed);
        return true;
    }
    return expected == (seen | kMailboxClosed);  // closed by the host with no new work
}

// Resident launch, lane 0 of a warp with nothing to trace: sleep 1, 2, 4, 8 us between
// polls (`waiting`: the last claim found nothing) so thousands of idle warps do not
// crowd the queue's cache lines, and after p.idle_us of sleep close the mailbox unless
// new work arrived.  True when the warp is to stop; every wait here is bounded.
__device__ __forceinline__ bool resident_wait(const BatchParams& p, ResidentWarp& rw, bool waiting) {
    if (rw.idle_ns >= p.idle_us * 1000u) {
        rw.idle_ns = 0;
        rw.sleep_ns = 1000;
        return resident_try_close(p, rw.pub_chunks, rw.pub_views);
    }
    if (waiting) {
        __nanosleep(rw.sleep_ns);
        rw.idle_ns += rw.sleep_ns;
        rw.sleep_ns = min(rw.sleep_ns * 2u, 8000u);
    }
    return false;
}

// Resident launch: `n` pixels of view `view` have stored all their records.  The
// caller's warp has synchronised after the stores; this lane's fence orders them (and,
// cumulatively, the other lanes') before the decrement, and the decrement that empties
// the count raises the view's done flag in host memory.
__device__ __forceinline__ void resident_pixels_done(const BatchParams& p, uint32_t view, uint32_t n) {
    __threadfence();
    if (atomicSub(p.remaining + view, n) == n) {
        __threadfence_system();
        *reinterpret_cast<volatile uint32_t*>(p.done_flags + view) = 1u;
    }
}

// Claims of a launch's queue.  A claim of its counter is a turn at one address for every warp of the
// chip at once, and with claims of half a tile a launch of few or short rays waits for little else.
// There (kOwn) a warp's first claim is its own number and the following come from the counter: two
// 640x360 GLSL views of a terrain 42.6 -> 40.0 us, two of 160x90 26.9 -> 24.8; of an empty world, where
// every ray leaves the grid in a few steps, 22.7 -> 20.6 (17.0 with whole tiles, and the terrain 46.9), and
// with 4 bounces 24.7 -> 22.7 (19.1 with whole tiles, and the terrain 194 for 168).  Where claims are
// whole tiles the counter is no limit, and neighbouring first claims for the warps of a block cost 44 M
// rays over 154 views 2 %.
__device__ __forceinline__ uint32_t warp_number() { return (blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
template <bool kOwn>
__device__ __forceinline__ uint32_t next_claim(const BatchParams& p) {
    return atomicAdd(p.queue, 1u) + (kOwn ? (gridDim.x * blockDim.x) >> 5 : 0u);
}

// kFull: the launch may hold views with the GPU renderer's whole path (a separate
// instantiation, so the others keep their code and registers).  64 registers (32 warps a SM)
// are enough for the CPU traversal (two 720p views of 4 bounces: 355 us against 382 us with
// 72 and 379 us with 56), not for the GLSL modes (two worlds' whole paths: 654 us against 626 us).
// kStall: rays that stand still (stalled) end early, looked at between the slices of a round.  A round
// lasts until half of its lanes have ended, and stalled lanes hold it up to the cap.  In the GLSL modes
// 35 to 41 % of a camera's primary rays stand still when it lies in the plane of an empty brick's face
// (of others none): there a 720p view of a terrain with 2 bounces 382 -> 152 us, anisotropic 358 ->
// 160; elsewhere the test costs up to 0.7 %, so stall_launch asks for it where some camera has a
// whole coordinate (a resident launch, whose views are not known, always looks).  Of views whose world
// origin is not near nearly all rays do (two such 720p views with sun rays, CPU traversal: 599 us in
// tile_kernel, 193 here; GLSL 1140 and 255).  In the CPU traversal of other views 1 ray in 500 does,
// and the test costs 6 % (spills).
template <bool kCount, bool kGlsl, bool kResident, bool kAniso, bool kFull, bool kStall>
__global__ void __maxnreg__(kGlsl ? 72 : 64) persistent_kernel(BatchParams p) {
    if constexpr (kAniso) fill_forward_lut();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    // warp-uniform queue state: rays [q_next, q_end) of view q_view
    uint32_t q_view = 0, q_next = 0, q_end = 0;
    bool q_empty = false, q_inside = false;  // q_inside: origin_inside_near() for q_view's camera
    // lane state
    bool active = false;
    // path: kind of the current ray (0 primary, then shadow or bounce number) in bits
    // 0-7, last kind of the pixel's path in bits 8-15, shadow flag in bit 16, ray
    // ended with its record pending in bit 17 (kEnded), that ray hit in bit 18 (kHit)
    constexpr uint32_t kEnded = 1u << 17, kHit = 1u << 18;
    uint32_t pixel = 0, path = 0, iter = 0, vidx = 0;
    RayState s;
    uint32_t rays = 0, hits = 0;
    TraceCounters cnt{0, 0};
    // resident launches: the warp's mailbox state and its count of finished pixels not
    // yet subtracted (lane 0)
    __shared__ ResidentWarp s_resident[16];  // warps_per_block <= 16 (checked when planning)
    ResidentWarp& rw = s_resident[threadIdx.x >> 5];
    if (kResident && lane == 0) rw = ResidentWarp{0, 0, kNoChunk, 0, 0, 1000, kNoView, 0, kNoView, 0};
    // resident launches: the entry of the view the warp takes rays from (q_view), so
    // that ray setup reads shared memory instead of making L2 round trips
    __shared__ ViewDev s_views[16];
    ViewDev& sview = s_views[threadIdx.x >> 5];
    // the GPU renderer's whole path: the hit frame (origin xyz, normal xyz) kept across a
    // sun ray, 6 floats per thread (dynamic shared memory, sized only for such batches)
    extern __shared__ float s_pend[];

    for (;;) {
        bool finished = false;  // a pixel's path ended this round (resident completion)
        // Rays that ended during the last DDA round are retired together here, so the
        // record store and the next ray of the path run once per round for all of
        // them instead of once per lane that happens to end on a given step.
        if (path & kEnded) {
            const bool hit = (path & kHit) != 0;
            path &= ~(kEnded | kHit);
            const ViewDev* v = p.views + vidx;
            const bool vs = kResident && vidx == rw.cached_view;
            if (vs) v = &sview;
            uint4* rec = p.out + vget<kResident>(&v->out_base, vs) + pixel;
            uint32_t kind = path & 0xFF;
            const uint32_t last_kind = (path >> 8) & 0xFF;
            const int4 wv = vs ? *reinterpret_cast<const int4*>(v->wo) : ldv<kResident>(reinterpret_cast<const int4*>(v->wo));
            const size_t plane = (size_t)vget<kResident>(&v->width, vs) * vget<kResident>(&v->height, vs);
            const DevWorld w = load_world(p.worlds + wv.w);
            rec[kind * plane] = pack_state<kGlsl>(s, hit_material(s, w.payload, hit), hit, iter, pixel);
            rays++;
            if (kCount && hit) hits++;
            // the GPU renderer's whole path goes on after a sun ray, hit or miss
            const bool full = kFull && (path & kPathFull) != 0, after_sun = full && full_is_sun(kind);
            if ((hit || after_sun) && kind < last_kind) {
                path++;
                kind++;
                float ox, oy, oz, dx, dy, dz;
                const float sun[3] = {vget<kResident>(&v->sun[0], vs), vget<kResident>(&v->sun[1], vs),
                                      vget<kResident>(&v->sun[2], vs)};
                if (full) {
                    // a sun ray starts from the hit just traced, whose frame is kept (shared
                    // memory, one slot per thread) for the bounce after it; a bounce after a
                    // sun ray starts from that kept frame, one after a bounce from its hit
                    float nx, ny, nz;
                    float* pend = s_pend + threadIdx.x;
                    const uint32_t bs = blockDim.x;
                    if (after_sun) {
                        ox = pend[0];
                        oy = pend[bs];
                        oz = pend[2 * bs];
                        nx = pend[3 * bs];
                        ny = pend[4 * bs];
                        nz = pend[5 * bs];
                    } else {
                        hit_frame<kGlsl>(s, ox, oy, oz, nx, ny, nz);
                    }
                    if (full_is_sun(kind)) {
                        pend[0] = ox;
                        pend[bs] = oy;
                        pend[2 * bs] = oz;
                        pend[3 * bs] = nx;
                        pend[4 * bs] = ny;
                        pend[5 * bs] = nz;
                        dx = sun[0];
                        dy = sun[1];
                        dz = sun[2];
                    } else {
                        bounce_dir(pixel, full_bounce(kind), nx, ny, nz, dx, dy, dz);
                    }
                } else {
                    next_path_ray<kGlsl>(s, ((path >> 16) & 1u) != 0, sun, pixel, kind, ox, oy, oz, dx, dy, dz);
                }
                const int32_t wo3[3] = {wv.x, wv.y, wv.z};
                ray_start<kGlsl>(s, clip_box(w, wo3), ox, oy, oz, dx, dy, dz, wv.x, wv.y, wv.z, kGlsl);
                iter = 0;
            } else {
                for (uint32_t kk = kind + 1; kk <= last_kind; kk++) rec[kk * plane] = no_ray_hit();
                active = false;
                finished = true;
            }
        }
        if (kResident) {
            // Finished pixels are counted per warp (rw.acc_n, of view rw.acc_view) and
            // subtracted from the view's remaining count once no lane of the warp
            // traces that view any more: one atomic per warp and stretch of a view,
            // not one per round (a large view would otherwise queue hundreds of
            // thousands of atomics on one counter).  Pixels of another view that end
            // meanwhile are subtracted at once.
            const uint32_t fm = __ballot_sync(0xffffffffu, finished);
            if (fm) {
                const uint32_t first = __shfl_sync(0xffffffffu, vidx, __ffs(fm) - 1);
                uint32_t av = 0;
                if (lane == 0) {
                    if (rw.acc_view == kNoView) rw.acc_view = first;
                    av = rw.acc_view;
                }
                av = __shfl_sync(0xffffffffu, av, 0);
                const uint32_t same = __ballot_sync(0xffffffffu, finished && vidx == av);
                if (lane == 0) rw.acc_n += (uint32_t)__popc(same);
                if (fm & ~same) {
                    __syncwarp();  // the records of every lane before the leader's fence
                    if (finished && vidx != av) {
                        const uint32_t peers = __match_any_sync(fm & ~same, vidx);
                        if (lane == (uint32_t)__ffs(peers) - 1u) resident_pixels_done(p, vidx, __popc(peers));
                    }
                }
            }
            const uint32_t av = __shfl_sync(0xffffffffu, lane == 0 ? rw.acc_view : 0u, 0);
            if (av != kNoView && !__any_sync(0xffffffffu, active && vidx == av)) {
                __syncwarp();
                if (lane == 0) {
                    resident_pixels_done(p, av, rw.acc_n);
                    rw.acc_view = kNoView;
                    rw.acc_n = 0;
                }
            }
        }
        // Compaction and regeneration: once fewer than p.refill lanes trace, the idle ones
        // take new rays from the warp's chunk.  With rounds as long as the iteration cap
        // (p.inner >= max_iters) a round ends only when every lane has finished, so the
        // warp takes 32 new rays of one tile together, which keeps camera rays coherent;
        // bounce rays, incoherent anyway, gain from refills in the middle of a path.
        const uint32_t act = __ballot_sync(0xffffffffu, active);
        bool q_wait = false;  // resident: nothing published right now
        if ((uint32_t)__popc(act) < p.refill && !q_empty) {
            uint32_t idle = kResident ? ~act : ~act & p.lanes;
            while (idle) {
                if (q_next >= q_end) {
                    uint32_t c = 0, nv = p.n_views, part = 0;
                    if (kResident) {
                        if (lane == 0) {
                            c = resident_claim(p, rw, act != 0);
                            nv = rw.pub_views;
                        }
                        c = __shfl_sync(0xffffffffu, c, 0);
                        nv = __shfl_sync(0xffffffffu, nv, 0);
                        if (c == kClaimStop) {
                            q_empty = true;
                            break;
                        }
                        if (c == kClaimEmpty) {
                            q_wait = true;
                            break;
                        }
                    } else {
                        if (q_end == 0) {
                            c = warp_number();
                        } else {
                            if (lane == 0) c = next_claim<true>(p);
                            c = __shfl_sync(0xffffffffu, c, 0);
                        }
                        part = c & ((1u << p.split_log2) - 1u);
                        c >>= p.split_log2;
                        if (c >= p.total_chunks) {
                            q_empty = true;
                            break;
                        }
                        c += p.chunk_first;
                    }
                    // a warp's claims only grow, so the chunk lies in view q_view or a
                    // later one: test the next view's start before searching
                    uint32_t lo = q_view, hi = nv;
                    if (lo + 1 < hi && ldv<kResident>(p.chunk_base + lo + 1) <= c)
                        lo++;
                    else
                        hi = lo + 1;
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (ldv<kResident>(p.chunk_base + mid) <= c)
                            lo = mid;
                        else
                            hi = mid;
                    }
                    q_view = lo;
                    q_next = (c - ldv<kResident>(p.chunk_base + lo)) * p.chunk_rays;
                    if (!kResident) q_next += part * (p.chunk_rays >> p.split_log2);
                    if (kResident && lo != rw.cached_view) {
                        // every lane is done with the old copy, and the loads below are
                        // ordered after lane 0's acquire of the hint that published lo
                        __syncwarp();
                        if (lane < sizeof(ViewDev) / 4)
                            reinterpret_cast<uint32_t*>(&sview)[lane] =
                                __ldcg(reinterpret_cast<const uint32_t*>(p.views + lo) + lane);
                        if (lane == 0) rw.cached_view = lo;
                        __syncwarp();
                    }
                    const ViewDev* qv = kResident ? &sview : p.views + lo;
                    q_end = min(q_next + (kResident ? p.chunk_rays : p.chunk_rays >> p.split_log2),
                                vget<kResident>(&qv->n_rays, true));
                    // the view's camera origin, shared by its rays: inside the clip box?
                    // (a resident view's world index is checked before it is used)
                    const int4 qwv = vget4<kResident>(reinterpret_cast<const int4*>(qv->wo));  // origin xyz, world
                    const int32_t qwo[3] = {qwv.x, qwv.y, qwv.z};
                    const bool inside = (!kResident || (uint32_t)qwv.w < p.n_worlds) &&
                                        origin_inside_near(clip_box(p.worlds[qwv.w], qwo), vget<kResident>(&qv->ox, true),
                                                           vget<kResident>(&qv->oy, true), vget<kResident>(&qv->oz, true));
                    if (kResident) {  // kept with the warp's other shared state (registers are short)
                        if (lane == 0) rw.q_inside = inside ? 1u : 0u;
                        __syncwarp();
                    } else {
                        q_inside = inside;
                    }
                    continue;
                }
                const uint32_t take = min(q_end - q_next, (uint32_t)__popc(idle));
                const uint32_t rank = __popc(idle & lt);
                const bool mine = ((idle >> lane) & 1u) && rank < take;
                const uint32_t assigned = __ballot_sync(0xffffffffu, mine);
                if (mine) {
                    const ViewDev* v = kResident ? &sview : p.views + q_view;
                    // width, height, tiles_x, tiles_x_magic
                    const uint4 geo = vget4<kResident>(reinterpret_cast<const uint4*>(&v->width));
                    const uint32_t r = q_next + rank;
                    const uint32_t t = r >> p.tile_size_log2, k = r & ((1u << p.tile_size_log2) - 1u);
                    uint32_t kx, ky;
                    if (p.morton) {
                        kx = compact_even_bits(k);
                        ky = compact_even_bits(k >> 1);
                    } else {
                        kx = k & ((1u << p.tile_w_log2) - 1u);
                        ky = k >> p.tile_w_log2;
                    }
                    const uint32_t tw = 1u << p.tile_w_log2, th = 1u << (p.tile_size_log2 - p.tile_w_log2);
                    // t / tiles_x by multiply-high: the estimate is the quotient or one more
                    uint32_t trow = geo.w ? __umulhi(t, geo.w) : t;
                    if (trow * geo.z > t) trow--;
                    const uint32_t px = (t - trow * geo.z) * tw + kx, py = trow * th + ky;
                    const uint32_t width = geo.x, height = geo.y;
                    bool valid = px < width && py < height;
                    const int4 wv = vget4<kResident>(reinterpret_cast<const int4*>(v->wo));  // origin xyz, world
                    const uint2 mp = vget4<kResident>(reinterpret_cast<const uint2*>(&v->max_iters));  // cap, path
                    if (kResident && valid) {
                        // a resident launch's views arrive while it runs: check what the
                        // ray would index (its world, its records) before touching it
                        const uint32_t kinds = 1u + ((mp.y >> 8) & 0xFFu);
                        valid = (uint32_t)wv.w < p.n_worlds &&
                                vget<kResident>(&v->out_base, true) + (unsigned long long)width * height * kinds <=
                                    p.out_records;
                    }
                    if (valid) {
                        vidx = q_view;
                        pixel = py * width + px;
                        iter = 0;
                        path = mp.y;
                        // d0, du, dv with the camera origin in the fourth lanes
                        const float4 g0 = vget4<kResident>(reinterpret_cast<const float4*>(v->d0));
                        const float4 g1 = vget4<kResident>(reinterpret_cast<const float4*>(v->du));
                        const float4 g2 = vget4<kResident>(reinterpret_cast<const float4*>(v->dv));
                        const float d0[3] = {g0.x, g0.y, g0.z}, du[3] = {g1.x, g1.y, g1.z}, dv[3] = {g2.x, g2.y, g2.z};
                        float dx, dy, dz;
                        camera_ray(d0, du, dv, px, py, dx, dy, dz);
                        const int32_t wo3[3] = {wv.x, wv.y, wv.z};
                        if (kResident ? rw.q_inside != 0 : q_inside)
                            ray_start_inside<kGlsl>(s, g0.w, g1.w, g2.w, dx, dy, dz, wv.x, wv.y, wv.z);
                        else
                            ray_start<kGlsl>(s, clip_box(load_world(p.worlds + wv.w), wo3), g0.w, g1.w, g2.w, dx, dy, dz,
                                             wv.x, wv.y, wv.z);
                        active = true;
                    }
                }
                idle &= ~assigned;
                q_next += take;
            }
        }
        if (__ballot_sync(0xffffffffu, active) == 0) {
            if (q_empty) break;
            if (kResident) {
                // nothing to trace and nothing published: wait for the host
                bool stop = false;
                if (lane == 0) stop = resident_wait(p, rw, q_wait);
                if (__shfl_sync(0xffffffffu, stop ? 1u : 0u, 0)) q_empty = true;
                continue;
            }
        }
        if (kResident && lane == 0 && rw.idle_ns) {
            rw.idle_ns = 0;
            rw.sleep_ns = 1000;
        }
        // GLSL mode: does any lane trace a shadow or bounce ray (rayCastCoarse's)?
        const bool any_coarse = kGlsl && __any_sync(0xffffffffu, active && (path & 0xFFu) != 0);
        // The lane's world origin, cap and world, read again for each round: held in registers
        // across the retirement and refill above they cost the step loop spills.
        int4 wv{};
        DevWorld w{};
        uint32_t max_iters = 0;
        if (active) {
            const ViewDev* v = p.views + vidx;
            if (kResident && vidx == rw.cached_view) {
                wv = *reinterpret_cast<const int4*>(sview.wo);
                max_iters = sview.max_iters;
            } else {
                wv = ldv<kResident>(reinterpret_cast<const int4*>(v->wo));
                max_iters = ldv<kResident>(&v->max_iters);
            }
            if (kGlsl && (path & 0xFFu)) max_iters = min(max_iters, kCoarseMaxIters);  // rayCastCoarse's cap
            w = load_world(p.worlds + wv.w);
        }
        // Steps until half the tracing lanes have ended, in slices of p.inner: the lanes left
        // keep the warp busy, and enough have ended to share a retirement.  Two 720p views of
        // 4 bounces: 372 us, five eighths left 374 us, three eighths 377 us.
        const uint32_t stop = (uint32_t)__popc(__ballot_sync(0xffffffffu, active)) / 2u;
        float t0 = no_t();
        do {
            if (active && !(path & kEnded)) {
                const uint32_t kmax = min(p.inner, max_iters - iter);  // an active lane has iter < max_iters
                uint32_t k = 0;
                // GLSL mode: the rayCastCoarse variant while some lane traces a shadow or
                // bounce ray, the anisotropic one for views that ask for it
                const uint32_t st = dda_steps_mode<kCount, kGlsl, true>(s, w, wv.x, wv.y, wv.z, cnt, any_coarse,
                                                                  (path & 0xFFu) != 0, kAniso, iter, k, kmax);
                if constexpr (kStall) {  // (the counting launch takes every step)
                    if (st == kStepContinue && stalled<kGlsl>(s, t0, (path & 0xFFu) != 0, iter)) iter = max_iters - k;
                    t0 = last_t<kGlsl>(s);
                }
                iter += k;  // the iteration a ray left on, or max_iters when the cap ran out
                if (st != kStepContinue)
                    path |= kEnded | (st == kStepHit ? kHit : 0u);
                else if (iter >= max_iters)
                    path |= kEnded;
            }
        } while ((uint32_t)__popc(__ballot_sync(0xffffffffu, active && !(path & kEnded))) > stop);
    }
    // warp totals, one atomic per warp
    for (int off = 16; off > 0; off >>= 1) {
        rays += __shfl_xor_sync(0xffffffffu, rays, off);
        if (kCount) {
            hits += __shfl_xor_sync(0xffffffffu, hits, off);
            cnt.step_calls += __shfl_xor_sync(0xffffffffu, cnt.step_calls, off);
            cnt.occ_fetches += __shfl_xor_sync(0xffffffffu, cnt.occ_fetches, off);
        }
    }
    if (lane == 0) {
        atomicAdd(p.counters + 0, (unsigned long long)rays);
        if (kCount) {
            atomicAdd(p.counters + 1, (unsigned long long)cnt.step_calls);
            atomicAdd(p.counters + 2, (unsigned long long)cnt.occ_fetches);
            atomicAdd(p.counters + 3, (unsigned long long)hits);
        }
    }
}

// Launches whose views have no bounces (primary rays, or primary and one sun ray): each warp
// claims a chunk of tiles and traces it 32 rays at a time, a pixel's rays per lane
// (trace_pixel) before it takes the next 32.  Bound by instruction issue.  Neighbouring camera
// rays are of a length (92-96 % of lanes busy in an 8x4 group on terrain), so nothing is
// gained by refilling lanes one by one, and without it the view, its world and what its rays
// share (ViewStart) belong to the warp: in shared memory, read at a ray's start, the step
// loop's part in registers.  Warp instructions for 32 primary rays (smsp__inst_executed at caps of
// 1 and 5 steps): 228 and 47 to 49 a step (335 and 52 in the persistent kernel when this one was
// built), and 175 in all for a camera in a solid voxel.
// 44 M rays over 154 views of 16 mixed worlds: 701 us against 1109 us, 658 us with the packed adds
// and 64 registers; six 1080p terrain views with sun rays: 754 us against 1035 us, 718 us.  64
// registers, 32 warps a SM, in the CPU traversal (72, 28 warps: 670 and 740 us, 56: 714 and 767);
// 72 in the GLSL modes (64 cost an anisotropic 1800x1800 batch 9 %).
// kPacked: the records are stored in the 12-byte form.  kSplit: claims are parts of a tile
// (launch_persistent), an instantiation of its own as their arithmetic cost the others 0.5 %.
template <bool kGlsl, bool kAniso, bool kPacked, bool kSplit>
__global__ void __maxnreg__(kGlsl ? 72 : 64) tile_kernel(BatchParams p) {
    if constexpr (kAniso) fill_forward_lut();
    // what the warp's view needs at a ray's start (warps_per_block <= 16)
    struct Warp {
        ViewDev v;
        DevWorld w;
        ViewStart start;
    };
    __shared__ Warp s_warps[16];
    Warp& sw = s_warps[threadIdx.x >> 5];
    const ViewDev& v = sw.v;
    DevWorld w{};  // a copy in registers: the step loop reads its table addresses and strides
    const uint32_t lane = threadIdx.x & 31;
    // the lane's pixel in a tile's first 32 (the next 32 lie `rows` rows below), or in the part of a
    // tile that the warp has claimed (split_log2 > 0); outside every view where the lane has none
    uint32_t kx = 0, ky = 0;
    const auto place = [&](uint32_t first) {
        const uint32_t k = first + lane;
        if (p.morton) {
            kx = compact_even_bits(k);
            ky = compact_even_bits(k >> 1);
        } else {
            kx = k & ((1u << p.tile_w_log2) - 1u);
            ky = k >> p.tile_w_log2;
        }
        if (kSplit && !((p.lanes >> lane) & 1u)) kx = 1u << 16;
    };
    place(0);
    const uint32_t tile_h = 1u << (p.tile_size_log2 - p.tile_w_log2), rows = kSplit ? tile_h : 32u >> p.tile_w_log2;
    const uint32_t chunk_tiles = p.chunk_rays >> p.tile_size_log2;
    uint32_t view = 0, loaded = kNoView, rays = 0;
    uint32_t claim = kSplit ? warp_number() : __shfl_sync(0xffffffffu, lane == 0 ? next_claim<false>(p) : 0u, 0);
    for (;;) {
        uint32_t c = claim;
        if (kSplit) {
            place((c & ((1u << p.split_log2) - 1u)) << (p.tile_size_log2 - p.split_log2));
            c >>= p.split_log2;
        }
        if (c >= p.total_chunks) break;
        c += p.chunk_first;
        // a warp's claims only grow, so the chunk lies in the last view or a later one
        uint32_t hi = p.n_views;
        if (view + 1 < hi && __ldg(p.chunk_base + view + 1) <= c)
            view++;
        else
            hi = view + 1;
        while (hi - view > 1) {
            const uint32_t mid = (view + hi) >> 1;
            if (__ldg(p.chunk_base + mid) <= c)
                view = mid;
            else
                hi = mid;
        }
        if (view != loaded) {
            loaded = view;
            __syncwarp();
            reinterpret_cast<uint32_t*>(&sw.v)[lane] = __ldg(reinterpret_cast<const uint32_t*>(p.views + view) + lane);
            const uint32_t wi = __ldg(&p.views[view].world);
            if (lane < sizeof(DevWorld) / 4)
                reinterpret_cast<uint32_t*>(&sw.w)[lane] = __ldg(reinterpret_cast<const uint32_t*>(p.worlds + wi) + lane);
            __syncwarp();
            w = sw.w;
            ViewStart vs = view_start(w, v);
            if (!kGlsl && vs.inside) {
                // iteration 0 of every ray of the view: the table entry and code at the origin
                const uint32_t x = (uint32_t)(v.wo[0] + __float2int_rd(v.ox)),
                               y = (uint32_t)(v.wo[1] + __float2int_rd(v.oy)),
                               z = (uint32_t)(v.wo[2] + __float2int_rd(v.oz));
                const uint32_t e = __ldg(w.bricks + (x >> 3) + (z >> 3) * w.bsx + (y >> 3) * w.bsxz);
                if (e < kBrickEmpty) {
                    const size_t at = (size_t)e * 512 + ((x & 7u) | (z & 7u) << 3 | (y & 7u) << 6);
                    const uint32_t code = __ldg(w.codes + at);
                    vs.mask = code == kCodeSolid ? kStartSolid : code;
                    vs.material = __ldg(w.payload + at);
                } else {
                    vs.mask = e & 31u;
                }
                vs.voxel[0] = x + kVoxelBias;
                vs.voxel[1] = y + kVoxelBias;
                vs.voxel[2] = z + kVoxelBias;
            }
            if (lane == 0) sw.start = vs;
            __syncwarp();
        }
        uint32_t t = (c - v.chunk_base) * chunk_tiles;
        const uint32_t t_end = min(t + chunk_tiles, v.n_rays >> p.tile_size_log2);
        uint32_t ty = v.tiles_x_magic ? __umulhi(t, v.tiles_x_magic) : t;
        if (ty * v.tiles_x > t) ty--;
        uint32_t tx = t - ty * v.tiles_x;
        uint32_t y = ty * tile_h;
        for (;;) {
            const uint32_t px = (tx << p.tile_w_log2) + kx, py = y + ky;
            if (px < v.width && py < v.height)
                rays += trace_pixel<kGlsl, kAniso, false, kPacked>(v, w, sw.start, px, py, p.out);
            __syncwarp();
            y += rows;
            if ((y & (tile_h - 1u)) == 0) {  // the tile is done
                if (++t == t_end) break;
                y -= tile_h;
                if (++tx == v.tiles_x) {
                    tx = 0;
                    y += tile_h;
                }
            }
        }
        claim = __shfl_sync(0xffffffffu, lane == 0 ? next_claim<kSplit>(p) : 0u, 0);
    }
    for (int off = 16; off > 0; off >>= 1) rays += __shfl_xor_sync(0xffffffffu, rays, off);
    if (lane == 0) atomicAdd(p.counters, (unsigned long long)rays);
}

uint32_t log2u(uint32_t v) {
    uint32_t r = 0;
    while ((1u << r) < v) r++;
    return r;
}

}  // namespace

void set_view_camera(ViewDev& d, const vrt_camera& c) {
    for (int k = 0; k < 3; k++) {
        d.d0[k] = c.d0[k];
        d.du[k] = c.du[k];
        d.dv[k] = c.dv[k];
        d.wo[k] = c.world_origin[k];
    }
    d.ox = c.origin[0];
    d.oy = c.origin[1];
    d.oz = c.origin[2];
    d.width = c.width;
    d.height = c.height;
}

ViewDev make_view_dev(const vrt_view& v) {
    ViewDev d{};
    set_view_camera(d, v.cam);
    d.world = v.world;
    d.max_iters = eff_iters(v.max_iters, view_glsl(v));
    d.aniso = view_aniso(v) ? 1u : 0u;
    const uint32_t shadow = (v.flags & VRT_VIEW_SHADOW) ? 1u : 0u;
    if (shadow && v.n_bounces)  // the GPU renderer's whole path: sun rays among the bounces
        d.path = (uint32_t)(view_record_count(v) / ((uint64_t)v.cam.width * v.cam.height) - 1) << 8 | kPathFull;
    else
        d.path = (shadow ? 1u : v.n_bounces) << 8 | shadow << 16;
    for (int c = 0; c < 3; c++) d.sun[c] = v.sun_dir[c];
    return d;
}

namespace {

using ViewPathFn = void (*)(DevWorld, ViewDev, ViewStart, uint32_t, uint4*);
template <bool kBounces, bool kThin, bool kFar = false>
ViewPathFn view_path_fn(bool glsl, bool aniso) {
    if (glsl && aniso) return view_path_kernel<true, true, kBounces, kThin, kFar>;
    if (glsl) return view_path_kernel<true, false, kBounces, kThin, kFar>;
    return view_path_kernel<false, false, kBounces, kThin, kFar>;
}

vrt_status launch_view_path(vrt_world* w, const ViewDev& v, bool glsl, vrt_hit* hits, cudaStream_t stream) {
    const bool far = !near_origin(v.wo);
    const uint32_t ll = far ? 5u : thin_lanes_log2((uint64_t)v.width * v.height, sm_count());
    const dim3 grid = thin_grid(ll, v.width, v.height);
    L2Window l2;
    vrt_status st = l2.enter(w, stream);
    if (st != VRT_OK) return st;
    uint4* out = reinterpret_cast<uint4*>(hits);
    const DevWorld dw = w->dev();
    const ViewStart vs = view_start(dw, v);
    const bool bounces = v.last_kind() > 1u || (v.last_kind() == 1u && !v.shadow());
    const auto fn = far       ? view_path_fn<true, false, true>
                    : bounces ? (ll < 5 ? view_path_fn<true, true> : view_path_fn<true, false>)
                              : (ll < 5 ? view_path_fn<false, true> : view_path_fn<false, false>);
    const ViewPathFn kernel = fn(glsl, v.aniso);
    kernel<<<grid, kFrameThreads, 0, stream>>>(dw, v, vs, ll, out);
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

}  // namespace

uint32_t eff_iters(uint32_t m, bool glsl) {
    if (m == 0) return glsl ? VRT_GLSL_MAX_ITERS : VRT_DEFAULT_MAX_ITERS;
    return m > 65535u ? 65535u : m;
}

vrt_status check_same_mode(const vrt_view* views, uint32_t n) {
    for (uint32_t i = 1; i < n; i++)
        if (view_mode(views[i]) != view_mode(views[0])) {
            set_error("the views of one launch must share one traversal mode (VRT_VIEW_GLSL, VRT_VIEW_GLSL_ANISO)");
            return VRT_ERR_INVALID_ARG;
        }
    return VRT_OK;
}

vrt_status check_view(const vrt_view* v) {
    if (!v || v->cam.width == 0 || v->cam.height == 0 || v->cam.width > 16384 || v->cam.height > 16384 ||
        v->n_bounces > VRT_MAX_BOUNCES || (v->flags & ~(VRT_VIEW_SHADOW | VRT_VIEW_GLSL | VRT_VIEW_GLSL_ANISO)) ||
        ((v->flags & VRT_VIEW_GLSL_ANISO) && !(v->flags & VRT_VIEW_GLSL)) || !world_origin_ok(v->cam.world_origin)) {
        set_error("bad view: camera 1..16384 px, |world origin| <= 2^30, n_bounces <= 15, anisotropic LODs only "
                  "with the GLSL mode");
        return VRT_ERR_INVALID_ARG;
    }
    return VRT_OK;
}

uint64_t view_record_count(const vrt_view& v) {
    const uint64_t n = v.n_bounces;
    // primary; shadow; bounces; or the renderer's path: sun, bounces, sun after the first two
    const uint64_t kinds = 1 + ((v.flags & VRT_VIEW_SHADOW) ? (n ? 1 + n + std::min<uint64_t>(n, 2) : 1) : n);
    return kinds * v.cam.width * v.cam.height;
}

vrt_status normalize_batch_config(const vrt_batch_config* in, vrt_batch_config& cfg) {
    cfg = in ? *in : vrt_batch_config{};
    if (cfg.tile_w == 0 && cfg.tile_h == 0) cfg.tile_w = 8, cfg.tile_h = 8;
    const bool shape_ok = (cfg.tile_w == 8 && cfg.tile_h == 8) || (cfg.tile_w == 16 && cfg.tile_h == 4) ||
                          (cfg.tile_w == 32 && cfg.tile_h == 1);
    if (!shape_ok || (cfg.morton && cfg.tile_w != 8)) {
        set_error("tile must be 8x8 (optionally Morton), 16x4 or 32x1");
        return VRT_ERR_INVALID_ARG;
    }
    if (cfg.warps_per_block == 0) cfg.warps_per_block = 4;
    // refill_threshold 0 and chunk_tiles 0 stay 0: resolve_batch_defaults picks them from
    // the launch's views and grid
    if (cfg.inner_iters == 0) cfg.inner_iters = 16;
    if (cfg.warps_per_block > 16 || cfg.refill_threshold > 32 || cfg.chunk_tiles > 64 || cfg.inner_iters > 1024) {
        set_error("batch config out of range");
        return VRT_ERR_INVALID_ARG;
    }
    return VRT_OK;
}

uint32_t auto_chunk_tiles(uint64_t tiles, uint64_t warps) {
    if (warps == 0) return 1;
    return (uint32_t)std::min<uint64_t>(16, std::max<uint64_t>(1, tiles / (warps * 8)));
}

// Tiles per claim of tile_kernel where the config leaves it open, at most: the launch ends with
// the last claims, and 16 tiles (1,024 rays) of long rays run on for a third of a millisecond
// after the queue is empty (44 M rays over 154 views: 1466 us with 16 tiles, 1041 with 4, 968
// with 2, 950 with 1 in the kernel's first build; 658 with 2, 782 with 1 in the present one).
// The cap holds at every size, though where the tiles are many and their rays short more are better:
// 353 M rays of the same kind, half of whose views end at once, take 2.62 ms with 8 tiles and 2.89
// with 2, so a large recurring batch is worth a config of its own (autotune.py).
// Pixels with a sun ray are twice the work, so one tile up to kOneTileWarps a warp (six 1080p
// views 718 -> 697 us).
constexpr uint32_t kTileChunk = 2, kOneTileWarps = 64;
bool tile_launch(const vrt_view* views, uint32_t n) {
    for (uint32_t i = 0; i < n; i++)
        if (views[i].n_bounces) return false;
    return !far_launch(views, n);
}
bool far_launch(const vrt_view* views, uint32_t n) {
    for (uint32_t i = 0; i < n; i++)
        if (!near_origin(views[i].cam.world_origin)) return true;
    return false;
}
bool stall_launch(const vrt_view* views, uint32_t n) {
    for (uint32_t i = 0; i < n; i++)
        for (int c = 0; c < 3; c++)
            if (view_glsl(views[i]) && views[i].cam.origin[c] == std::floor(views[i].cam.origin[c])) return true;
    return far_launch(views, n);
}

void resolve_batch_defaults(vrt_batch_config& cfg, const vrt_view* views, uint32_t n, uint64_t warps) {
    bool bounces = false;
    uint64_t tiles = 0;
    for (uint32_t i = 0; i < n; i++) {
        bounces |= views[i].n_bounces > 0;
        tiles += (uint64_t)((views[i].cam.width + cfg.tile_w - 1) / cfg.tile_w) *
                 ((views[i].cam.height + cfg.tile_h - 1) / cfg.tile_h);
    }
    if (cfg.refill_threshold == 0) cfg.refill_threshold = bounces ? 28 : 16;
    if (cfg.chunk_tiles == 0) cfg.chunk_tiles = bounces ? 1 : auto_chunk_tiles(tiles, warps);
}

void resolve_launch_config(vrt_batch_config& cfg, const vrt_view* views, uint32_t n, uint64_t warps) {
    const bool open = cfg.chunk_tiles == 0;
    resolve_batch_defaults(cfg, views, n, warps);
    if (!open || !tile_launch(views, n)) return;
    bool sun = false;
    uint64_t pixels = 0;
    for (uint32_t i = 0; i < n; i++) {
        sun |= (views[i].flags & VRT_VIEW_SHADOW) != 0;
        pixels += (uint64_t)views[i].cam.width * views[i].cam.height;
    }
    cfg.chunk_tiles = sun && pixels / 64 < kOneTileWarps * warps ? 1 : std::min(cfg.chunk_tiles, kTileChunk);
}

vrt_status plan_views(const vrt_view* views, uint32_t n, uint32_t n_worlds, const vrt_batch_config& cfg_in,
                      LaunchPlan& plan, uint64_t warps) {
    vrt_status st;
    for (uint32_t i = 0; i < n; i++) {
        if ((st = check_view(&views[i])) != VRT_OK) return st;
        if (views[i].world >= n_worlds) {
            set_error("view references a world outside the list");
            return VRT_ERR_INVALID_ARG;
        }
    }
    if ((st = check_same_mode(views, n)) != VRT_OK) return st;
    vrt_batch_config cfg = cfg_in;
    resolve_launch_config(cfg, views, n, warps);
    plan.glsl = n > 0 && view_glsl(views[0]);
    plan.aniso = n > 0 && view_aniso(views[0]);
    plan.full = false;
    for (uint32_t i = 0; i < n; i++) plan.full |= view_full_path(views[i]);
    plan.tiles = tile_launch(views, n);
    plan.stall = stall_launch(views, n);
    plan.cfg = cfg;
    plan.tile_w_log2 = log2u(cfg.tile_w);
    plan.tile_size_log2 = log2u(cfg.tile_w * cfg.tile_h);
    plan.views.resize(n);
    plan.chunk_base.resize(n + 1);
    uint64_t chunks = 0, records = 0;
    for (uint32_t i = 0; i < n; i++) {
        ViewDev d = make_view_dev(views[i]);
        const uint32_t tx = (d.width + cfg.tile_w - 1) / cfg.tile_w;
        const uint32_t ty = (d.height + cfg.tile_h - 1) / cfg.tile_h;
        const uint64_t tiles = (uint64_t)tx * ty;
        d.tiles_x = tx;
        d.tiles_x_magic = div_magic(tx);
        d.n_rays = (uint32_t)(tiles << plan.tile_size_log2);
        d.chunk_base = (uint32_t)chunks;
        d.out_base = records;
        plan.chunk_base[i] = (uint32_t)chunks;
        chunks += (tiles + cfg.chunk_tiles - 1) / cfg.chunk_tiles;
        records += view_record_count(views[i]);
        plan.views[i] = d;
        if (chunks >= 0xffffffffull) {
            set_error("batch too large");
            return VRT_ERR_INVALID_ARG;
        }
    }
    plan.chunk_base[n] = (uint32_t)chunks;
    plan.chunks = (uint32_t)chunks;
    plan.records = records;
    return VRT_OK;
}

namespace {

// The kernel a launch runs: tiles (no view has bounces), or the persistent kernel's
// instantiation: counting, traversal mode, resident, whole-path views.
using PersistentFn = void (*)(BatchParams);
template <bool kCount, bool kResident, bool kFull, bool kGlslStall, bool kCpuStall>
PersistentFn persistent_fn_mode(bool glsl, bool aniso) {
    if (glsl && aniso) return persistent_kernel<kCount, true, kResident, true, kFull, kGlslStall>;
    if (glsl) return persistent_kernel<kCount, true, kResident, false, kFull, kGlslStall>;
    return persistent_kernel<kCount, false, kResident, false, kFull, kCpuStall>;
}
template <bool kPacked, bool kSplit>
PersistentFn tile_fn(bool glsl, bool aniso) {
    return glsl ? (aniso ? tile_kernel<true, true, kPacked, kSplit> : tile_kernel<true, false, kPacked, kSplit>)
                : tile_kernel<false, false, kPacked, kSplit>;
}
PersistentFn persistent_fn(bool count, bool glsl, bool aniso, bool resident, bool full, bool tiles, bool stall) {
    if (tiles && !count && !resident) return tile_fn<false, false>(glsl, aniso);
    if (resident)  // (its views are not known yet)
        return full ? persistent_fn_mode<false, true, true, true, false>(glsl, aniso)
                    : persistent_fn_mode<false, true, false, true, false>(glsl, aniso);
    if (count)
        return full ? persistent_fn_mode<true, false, true, false, false>(glsl, aniso)
                    : persistent_fn_mode<true, false, false, false, false>(glsl, aniso);
    if (stall)
        return full ? persistent_fn_mode<false, false, true, true, true>(glsl, aniso)
                    : persistent_fn_mode<false, false, false, true, true>(glsl, aniso);
    return full ? persistent_fn_mode<false, false, true, false, false>(glsl, aniso)
                : persistent_fn_mode<false, false, false, false, false>(glsl, aniso);
}

// Resident blocks per SM of that kernel: the variants differ in registers and shared memory
// (the anisotropic LUT is 8 KB per block).
cudaError_t persistent_occupancy(int& occ, int threads, bool count, bool glsl, bool aniso, bool resident, bool full,
                                 bool tiles, bool stall) {
    const size_t smem = full ? (size_t)threads * 6 * sizeof(float) : 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &occ, persistent_fn(count, glsl, aniso, resident, full, tiles, stall), threads, smem);
}

}  // namespace

vrt_status persistent_grid(int device, const vrt_batch_config& cfg, bool count, bool glsl, bool aniso, bool resident,
                           bool full, bool tiles, bool stall, int& blocks, int& threads) {
    int sms = 0, occ = 0;
    threads = (int)cfg.warps_per_block * 32;
    VRT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    VRT_CUDA(persistent_occupancy(occ, threads, count, glsl, aniso, resident, full, tiles, stall));
    occ = std::max(occ, 1);
    const int per_sm = (!count && cfg.blocks_per_sm) ? std::min<int>((int)cfg.blocks_per_sm, occ) : occ;
    blocks = sms * per_sm;
    return VRT_OK;
}

BatchParams make_params(const LaunchPlan& plan, const DevWorld* worlds, const ViewDev* views,
                        const uint32_t* chunk_base, uint32_t* queue, vrt_hit* out) {
    BatchParams p{};
    p.worlds = worlds;
    p.views = views;
    p.chunk_base = chunk_base;
    p.n_views = (uint32_t)plan.views.size();
    p.total_chunks = plan.chunks;
    p.chunk_first = 0;
    p.queue = queue;
    p.counters = reinterpret_cast<unsigned long long*>(reinterpret_cast<uint8_t*>(queue) + 16);
    p.out = reinterpret_cast<uint4*>(out);
    p.tile_w_log2 = plan.tile_w_log2;
    p.tile_size_log2 = plan.tile_size_log2;
    p.morton = plan.cfg.morton;
    p.chunk_rays = plan.cfg.chunk_tiles << plan.tile_size_log2;
    // at least 1: a warp whose lanes are all idle must always claim (a resident warp learns
    // of the mailbox's close only through a claim)
    p.refill = std::max(1u, plan.cfg.refill_threshold);
    p.inner = std::max(1u, plan.cfg.inner_iters);  // a round must step, or no ray would progress
    p.glsl = plan.glsl ? 1u : 0u;
    p.aniso = plan.aniso ? 1u : 0u;
    p.full = plan.full ? 1u : 0u;
    p.tiles = plan.tiles ? 1u : 0u;
    p.stall = plan.stall ? 1u : 0u;
    return p;
}

vrt_status launch_resident(const BatchParams& p, int blocks, int threads, cudaStream_t stream) {
    const PersistentFn fn = persistent_fn(false, p.glsl != 0, p.aniso != 0, true, p.full != 0, false, false);
    fn<<<blocks, threads, pend_bytes(p, threads), stream>>>(p);
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

vrt_status launch_persistent(const BatchParams& p, int blocks, int threads, bool count, cudaStream_t stream,
                             size_t zero_bytes) {
    if (zero_bytes) VRT_CUDA(cudaMemsetAsync(p.queue, 0, zero_bytes, stream));
    const bool tiles = p.tiles && !count;
    BatchParams q = p;
    q.split_log2 = 0;
    q.lanes = 0xffffffffu;
    if (p.chunk_rays == 64 && p.tile_size_log2 == 6)
        q.split_log2 = claim_split_log2(p.total_chunks, !tiles, sm_count());
    if (q.split_log2) q.lanes >>= 32 - (64 >> q.split_log2);
    // no more warps than claims: each takes a turn at the queue's counter and returns (64x64 views
    // 13.3 -> 11.3 us from within a solid voxel, 35.7 -> 33.5 with 3 bounces of a terrain)
    const uint64_t claims = std::max<uint64_t>(1, (uint64_t)p.total_chunks << q.split_log2);
    blocks = (int)std::min<uint64_t>((uint64_t)blocks, (claims * 32 + threads - 1) / threads);
    const bool glsl = p.glsl != 0, aniso = p.aniso != 0;
    const auto tile = q.split_log2 ? (p.packed ? tile_fn<true, true> : tile_fn<false, true>)
                                   : (p.packed ? tile_fn<true, false> : tile_fn<false, false>);
    const PersistentFn fn = tiles ? tile(glsl, aniso)
                                  : persistent_fn(count, glsl, aniso, false, p.full != 0, false, p.stall != 0);
    fn<<<blocks, threads, pend_bytes(p, threads), stream>>>(q);
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

namespace {

// vrt_batch_run_packed of views with bounces (tile_kernel stores this form itself): records
// [0, n) of one part as 12-byte vrt_hit_packed, one thread per record (three 4-byte stores: a warp's
// stores cover 384 contiguous bytes); the 16-byte records are read once, so they are loaded as streaming
static_assert(sizeof(vrt_hit_packed) == 12 && sizeof(vrt_hit) == 16, "record sizes");
__global__ void __launch_bounds__(256)
    pack_records_kernel(const uint4* __restrict__ in, uint32_t* __restrict__ out, uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint4 r = __ldcs(in + i);
        out[3 * i] = r.x;
        out[3 * i + 1] = r.w == VRT_NO_RAY ? (r.y & 0xFFFF00FFu) | (VRT_PACKED_NO_RAY << 8) : r.y;
        out[3 * i + 2] = r.z;
    }
}

}  // namespace
}  // namespace vrt

using namespace vrt;

// Device block of a batch's queue counter and launch counters, and the parts of vrt_batch_run.
constexpr size_t kQueueBytes = 64;
constexpr uint64_t kMaxParts = 32;

struct vrt_batch {
    int device = 0;
    std::vector<vrt_world*> worlds;
    std::vector<vrt_view> views;
    LaunchPlan plan;
    std::vector<DevWorld> wtab;  // last uploaded world table
    int blocks = 0, threads = 0, blocks_count = 0, threads_count = 0;
    // device
    DevWorld* d_worlds = nullptr;
    ViewDev* d_views = nullptr;
    uint32_t* d_chunk_base = nullptr;
    uint32_t* d_queue = nullptr;  // queue counter, 4 u64 counters at byte 16, part counters at byte 64
    unsigned long long* d_counters = nullptr;
    cudaStream_t last_stream = nullptr;
    DevBuf d_out;     // record buffer of vrt_batch_run
    DevBuf d_packed;  // 12-byte records of vrt_batch_run_packed
    // vrt_batch_run: copies of finished parts overlap the traversal of later parts
    cudaStream_t copy_stream = nullptr;
    std::vector<cudaEvent_t> part_done;
    cudaEvent_t copies_done = nullptr;
    // graph
    cudaGraphExec_t graph_exec = nullptr;
    vrt_hit* graph_hits = nullptr;
    // the world whose brick table the batch's launches keep in L2: the batch's only
    // VRT_WORLD_L2_PERSIST world (a stream carries one access-policy window), or none
    vrt_world* l2_world = nullptr;
};

namespace {

vrt_status refresh_worlds(vrt_batch* b, cudaStream_t stream) {
    std::vector<DevWorld> t(b->worlds.size());
    for (size_t i = 0; i < t.size(); i++) t[i] = b->worlds[i]->dev();
    if (t.size() == b->wtab.size() && std::memcmp(t.data(), b->wtab.data(), t.size() * sizeof(DevWorld)) == 0)
        return VRT_OK;
    VRT_CUDA(cudaMemcpyAsync(b->d_worlds, t.data(), t.size() * sizeof(DevWorld), cudaMemcpyHostToDevice, stream));
    VRT_CUDA(cudaStreamSynchronize(stream));
    b->wtab = t;
    return VRT_OK;
}

vrt_status enqueue_batch(vrt_batch* b, vrt_hit* hits, cudaStream_t stream, bool count) {
    L2Window l2;
    vrt_status st = l2.enter(b->l2_world, stream);
    if (st != VRT_OK) return st;
    BatchParams p = make_params(b->plan, b->d_worlds, b->d_views, b->d_chunk_base, b->d_queue, hits);
    return count ? launch_persistent(p, b->blocks_count, b->threads_count, true, stream)
                 : launch_persistent(p, b->blocks, b->threads, false, stream);
}

}  // namespace

extern "C" {

uint64_t vrt_view_records(const vrt_view* v) { return check_view(v) == VRT_OK ? view_record_count(*v) : 0; }

vrt_status vrt_render_path_device(vrt_world* w, const vrt_view* view, vrt_hit* hits, void* stream) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK || (st = check_view(view)) != VRT_OK) return st;
    if (!hits) {
        set_error("null hit buffer");
        return VRT_ERR_INVALID_ARG;
    }
    ViewDev d = make_view_dev(*view);
    d.out_base = 0;
    return launch_view_path(w, d, view_glsl(*view), hits, (cudaStream_t)stream);
}

vrt_status vrt_render_path(vrt_world* w, const vrt_view* view, vrt_hit* hits, void* stream_) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK || (st = check_view(view)) != VRT_OK) return st;
    if (!hits) {
        set_error("null hit buffer");
        return VRT_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(w->mu);
    cudaStream_t stream = (cudaStream_t)stream_;
    const size_t hb = view_record_count(*view) * sizeof(vrt_hit);
    VRT_CUDA(w->d_io.reserve(hb));
    ViewDev d = make_view_dev(*view);
    if ((st = launch_view_path(w, d, view_glsl(*view), (vrt_hit*)w->d_io.ptr, stream)) != VRT_OK) return st;
    VRT_CUDA(cudaMemcpyAsync(hits, w->d_io.ptr, hb, cudaMemcpyDeviceToHost, stream));
    VRT_CUDA(cudaStreamSynchronize(stream));
    return VRT_OK;
}

vrt_status vrt_batch_create(vrt_world* const* worlds, uint32_t n_worlds, const vrt_view* views, uint32_t n_views,
                            const vrt_batch_config* cfg_in, vrt_batch** out) {
    if (!out || !worlds || n_worlds == 0 || !views || n_views == 0) {
        set_error("batch needs worlds and views");
        return VRT_ERR_INVALID_ARG;
    }
    *out = nullptr;
    vrt_batch_config cfg;
    vrt_status st = normalize_batch_config(cfg_in, cfg);
    if (st != VRT_OK) return st;
    for (uint32_t i = 0; i < n_worlds; i++)
        if (!worlds[i] || worlds[i]->device != worlds[0]->device) {
            set_error("worlds must be non-null and on one device");
            return VRT_ERR_INVALID_ARG;
        }
    DeviceScope ds;
    VRT_CUDA(ds.enter(worlds[0]->device));
    // the launch grid first: an auto chunk size depends on the number of warps
    int grid_blocks = 0, grid_threads = 0;
    {
        bool full = false;
        for (uint32_t i = 0; i < n_views; i++) full |= view_full_path(views[i]);
        if ((st = persistent_grid(worlds[0]->device, cfg, false, view_glsl(views[0]), view_aniso(views[0]), false,
                                  full, tile_launch(views, n_views), stall_launch(views, n_views), grid_blocks,
                                  grid_threads)) != VRT_OK)
            return st;
    }
    auto* b = new vrt_batch;
    if ((st = plan_views(views, n_views, n_worlds, cfg, b->plan, (uint64_t)grid_blocks * (grid_threads / 32))) !=
        VRT_OK) {
        delete b;
        return st;
    }
    cfg = b->plan.cfg;
    b->device = worlds[0]->device;
    b->worlds.assign(worlds, worlds + n_worlds);
    uint32_t n_l2 = 0;
    for (uint32_t i = 0; i < n_worlds; i++)
        if (worlds[i]->flags & VRT_WORLD_L2_PERSIST) {
            n_l2++;
            b->l2_world = worlds[i];
        }
    if (n_l2 != 1) b->l2_world = nullptr;
    b->views.assign(views, views + n_views);
    auto fail = [&](vrt_status s) {
        vrt_batch_destroy(b);
        return s;
    };
    cudaError_t e = cudaMalloc(&b->d_worlds, sizeof(DevWorld) * n_worlds);
    if (e == cudaSuccess) e = cudaMalloc(&b->d_views, sizeof(ViewDev) * n_views);
    if (e == cudaSuccess) e = cudaMalloc(&b->d_chunk_base, sizeof(uint32_t) * (n_views + 1));
    if (e == cudaSuccess) e = cudaMalloc(&b->d_queue, kQueueBytes + kMaxParts * sizeof(uint32_t));
    if (e == cudaSuccess)
        e = cudaMemcpy(b->d_views, b->plan.views.data(), sizeof(ViewDev) * n_views, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(b->d_chunk_base, b->plan.chunk_base.data(), sizeof(uint32_t) * (n_views + 1),
                       cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail(cuda_fail(e, "batch allocation"));
    b->d_counters = reinterpret_cast<unsigned long long*>(reinterpret_cast<uint8_t*>(b->d_queue) + 16);
    if ((st = refresh_worlds(b, 0)) != VRT_OK) return fail(st);
    const bool glsl = b->plan.glsl, aniso = b->plan.aniso, full = b->plan.full;
    if ((st = persistent_grid(b->device, cfg, false, glsl, aniso, false, full, b->plan.tiles, b->plan.stall, b->blocks,
                              b->threads)) != VRT_OK)
        return fail(st);
    if ((st = persistent_grid(b->device, cfg, true, glsl, aniso, false, full, false, false, b->blocks_count,
                              b->threads_count)) != VRT_OK)
        return fail(st);
    *out = b;
    return VRT_OK;
}

vrt_status vrt_batch_destroy(vrt_batch* b) {
    if (!b) return VRT_OK;
    DeviceScope ds;
    ds.enter(b->device);
    cudaDeviceSynchronize();
    if (b->graph_exec) cudaGraphExecDestroy(b->graph_exec);
    for (cudaEvent_t e : b->part_done) cudaEventDestroy(e);
    if (b->copies_done) cudaEventDestroy(b->copies_done);
    if (b->copy_stream) cudaStreamDestroy(b->copy_stream);
    if (b->d_worlds) cudaFree(b->d_worlds);
    if (b->d_views) cudaFree(b->d_views);
    if (b->d_chunk_base) cudaFree(b->d_chunk_base);
    if (b->d_queue) cudaFree(b->d_queue);
    b->d_out.release();
    b->d_packed.release();
    delete b;
    return VRT_OK;
}

vrt_status vrt_batch_output_layout(const vrt_batch* b, uint64_t* offsets) {
    if (!b || !offsets) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    for (size_t i = 0; i < b->plan.views.size(); i++) offsets[i] = b->plan.views[i].out_base;
    offsets[b->plan.views.size()] = b->plan.records;
    return VRT_OK;
}

vrt_status vrt_batch_update_cameras(vrt_batch* b, const vrt_camera* cams, void* stream_) {
    if (!b || !cams) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    for (size_t i = 0; i < b->plan.views.size(); i++) {
        if (cams[i].width != b->plan.views[i].width || cams[i].height != b->plan.views[i].height) {
            set_error("camera resolution differs from the batch's view");
            return VRT_ERR_INVALID_ARG;
        }
        if (!world_origin_ok(cams[i].world_origin)) {
            set_error("camera world origin outside +-2^30");
            return VRT_ERR_INVALID_ARG;
        }
    }
    DeviceScope ds;
    VRT_CUDA(ds.enter(b->device));
    for (size_t i = 0; i < b->plan.views.size(); i++) {
        set_view_camera(b->plan.views[i], cams[i]);
        b->views[i].cam = cams[i];
    }
    cudaStream_t stream = (cudaStream_t)stream_;
    VRT_CUDA(cudaMemcpyAsync(b->d_views, b->plan.views.data(), sizeof(ViewDev) * b->plan.views.size(), cudaMemcpyHostToDevice,
                             stream));
    VRT_CUDA(cudaStreamSynchronize(stream));
    return VRT_OK;
}

vrt_status vrt_batch_launch(vrt_batch* b, vrt_hit* hits, void* stream_) {
    if (!b || !hits) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    DeviceScope ds;
    VRT_CUDA(ds.enter(b->device));
    cudaStream_t stream = (cudaStream_t)stream_;
    vrt_status st = refresh_worlds(b, stream);
    if (st != VRT_OK) return st;
    b->last_stream = stream;
    return enqueue_batch(b, hits, stream, false);
}

vrt_status vrt_batch_launch_graph(vrt_batch* b, vrt_hit* hits, void* stream_) {
    if (!b || !hits) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    DeviceScope ds;
    VRT_CUDA(ds.enter(b->device));
    cudaStream_t stream = (cudaStream_t)stream_;
    vrt_status st = refresh_worlds(b, stream);
    if (st != VRT_OK) return st;
    if (!b->graph_exec || b->graph_hits != hits) {
        if (b->graph_exec) {
            cudaGraphExecDestroy(b->graph_exec);
            b->graph_exec = nullptr;
        }
        cudaStream_t cap;
        VRT_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            st = enqueue_batch(b, hits, cap, false);
            e = cudaStreamEndCapture(cap, &g);
        }
        if (e == cudaSuccess && st == VRT_OK) e = cudaGraphInstantiate(&b->graph_exec, g, 0);
        if (g) cudaGraphDestroy(g);
        cudaStreamDestroy(cap);
        if (st != VRT_OK) return st;
        if (e != cudaSuccess) return cuda_fail(e, "capture batch graph");
        b->graph_hits = hits;
    }
    b->last_stream = stream;
    VRT_CUDA(cudaGraphLaunch(b->graph_exec, stream));
    return VRT_OK;
}

vrt_status vrt_batch_launch_per_view(vrt_batch* b, vrt_hit* hits, void* stream_) {
    if (!b || !hits) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    DeviceScope ds;
    VRT_CUDA(ds.enter(b->device));
    cudaStream_t stream = (cudaStream_t)stream_;
    for (size_t i = 0; i < b->plan.views.size(); i++) {
        vrt_status st =
            launch_view_path(b->worlds[b->plan.views[i].world], b->plan.views[i], b->plan.glsl, hits, stream);
        if (st != VRT_OK) return st;
    }
    b->last_stream = stream;
    return VRT_OK;
}

}  // extern "C"

namespace {

// vrt_batch_run and vrt_batch_run_packed: trace, (pack,) and copy to `host` part by part.
uint64_t part_count(uint64_t records) {
    uint64_t n = 1;
    while (n < kMaxParts && (n + 1) * (n + 1) << 18 <= records) n++;
    return n;
}

vrt_status run_parts(vrt_batch* b, void* host, bool packed, cudaStream_t stream) {
    DeviceScope ds;
    VRT_CUDA(ds.enter(b->device));
    const LaunchPlan& plan = b->plan;
    const size_t nv = plan.views.size();
    const bool direct = packed && plan.tiles;  // the kernel stores packed records itself
    if (!direct) VRT_CUDA(b->d_out.reserve(plan.records * sizeof(vrt_hit)));
    if (packed) VRT_CUDA(b->d_packed.reserve(plan.records * sizeof(vrt_hit_packed)));
    vrt_status st = refresh_worlds(b, stream);
    if (st != VRT_OK) return st;
    // Views are split into parts of about equal record count, at view boundaries.
    // All parts are launched first, one after another on `stream`; the copy of a
    // part's records (one contiguous range) waits for that part only, so the host
    // transfer of finished parts overlaps the traversal of the later ones.  More parts start
    // the copies earlier, but each launch ramps up and runs out (20-100 us): the best number
    // grows with the root of the batch.  Times on GB300 for views of mixed worlds, 12-byte
    // records, by parts: 3.0 M records 287 us (1), 249 (4); 9.3 M 655 (5), 662 (11), 695 (23);
    // 24.6 M 1705 (7), 1760 (15), 2088 (32); 353 M as ever 32.
    const uint64_t want = part_count(plan.records);
    std::vector<size_t> cut{0};
    for (size_t i = 1; i < nv; i++)
        if (plan.views[i].out_base * want >= plan.records * cut.size()) cut.push_back(i);
    cut.push_back(nv);
    const size_t parts = cut.size() - 1;
    if (!b->copy_stream) {
        VRT_CUDA(cudaStreamCreateWithFlags(&b->copy_stream, cudaStreamNonBlocking));
        VRT_CUDA(cudaEventCreateWithFlags(&b->copies_done, cudaEventDisableTiming));
    }
    while (b->part_done.size() < parts) {
        cudaEvent_t e;
        VRT_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        b->part_done.push_back(e);
    }
    auto first_record = [&](size_t v) { return v < nv ? plan.views[v].out_base : plan.records; };
    const uint4* d_full = (const uint4*)b->d_out.ptr;
    uint32_t* d_pack = (uint32_t*)b->d_packed.ptr;
    L2Window l2;
    if ((st = l2.enter(b->l2_world, stream)) != VRT_OK) return st;
    VRT_CUDA(cudaMemsetAsync(b->d_queue, 0, kQueueBytes + parts * sizeof(uint32_t), stream));
    for (size_t k = 0; k < parts; k++) {
        const size_t a = cut[k], e = cut[k + 1];
        BatchParams p = make_params(plan, b->d_worlds, b->d_views, b->d_chunk_base, b->d_queue,
                                    (vrt_hit*)(direct ? b->d_packed.ptr : b->d_out.ptr));
        p.queue = b->d_queue + kQueueBytes / sizeof(uint32_t) + k;
        p.packed = direct ? 1u : 0u;
        p.views = b->d_views + a;
        p.chunk_base = b->d_chunk_base + a;
        p.n_views = (uint32_t)(e - a);
        p.chunk_first = plan.chunk_base[a];
        p.total_chunks = plan.chunk_base[e] - plan.chunk_base[a];
        if ((st = launch_persistent(p, b->blocks, b->threads, false, stream, 0)) != VRT_OK) return st;
        const uint64_t r0 = first_record(a), n = first_record(e) - r0;
        if (packed && !direct && n) {
            const uint32_t blocks = (uint32_t)std::min<uint64_t>((n + 255) / 256, 4096);
            pack_records_kernel<<<blocks, 256, 0, stream>>>(d_full + r0, d_pack + 3 * r0, n);
            VRT_CUDA(cudaGetLastError());
        }
        VRT_CUDA(cudaEventRecord(b->part_done[k], stream));
    }
    const size_t rec_bytes = packed ? sizeof(vrt_hit_packed) : sizeof(vrt_hit);
    const uint8_t* src = packed ? (const uint8_t*)d_pack : (const uint8_t*)d_full;
    for (size_t k = 0; k < parts; k++) {
        const uint64_t r0 = first_record(cut[k]), r1 = first_record(cut[k + 1]);
        VRT_CUDA(cudaStreamWaitEvent(b->copy_stream, b->part_done[k], 0));
        if (r1 > r0)
            VRT_CUDA(cudaMemcpyAsync((uint8_t*)host + r0 * rec_bytes, src + r0 * rec_bytes, (r1 - r0) * rec_bytes,
                                     cudaMemcpyDeviceToHost, b->copy_stream));
    }
    VRT_CUDA(cudaEventRecord(b->copies_done, b->copy_stream));
    VRT_CUDA(cudaStreamWaitEvent(stream, b->copies_done, 0));
    b->last_stream = stream;
    VRT_CUDA(cudaStreamSynchronize(stream));
    return VRT_OK;
}

}  // namespace

extern "C" {

vrt_status vrt_batch_run(vrt_batch* b, vrt_hit* hits_host, void* stream) {
    if (!b || !hits_host) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    return run_parts(b, hits_host, false, (cudaStream_t)stream);
}

vrt_status vrt_batch_run_packed(vrt_batch* b, vrt_hit_packed* records_host, void* stream) {
    if (!b || !records_host) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    return run_parts(b, records_host, true, (cudaStream_t)stream);
}

vrt_status vrt_batch_get_stats(vrt_batch* b, vrt_batch_stats* out) {
    if (!b || !out) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    DeviceScope ds;
    VRT_CUDA(ds.enter(b->device));
    VRT_CUDA(cudaStreamSynchronize(b->last_stream));
    unsigned long long c[4];
    VRT_CUDA(cudaMemcpy(c, b->d_counters, sizeof(c), cudaMemcpyDeviceToHost));
    out->rays_cast = c[0];
    out->step_calls = c[1];
    out->occ_fetches = c[2];
    out->hits = c[3];
    return VRT_OK;
}

vrt_status vrt_batch_measure(vrt_batch* b, vrt_hit* hits, void* stream_, vrt_batch_stats* out) {
    if (!b || !hits || !out) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    DeviceScope ds;
    VRT_CUDA(ds.enter(b->device));
    cudaStream_t stream = (cudaStream_t)stream_;
    vrt_status st = refresh_worlds(b, stream);
    if (st != VRT_OK || (st = enqueue_batch(b, hits, stream, true)) != VRT_OK) return st;
    b->last_stream = stream;
    return vrt_batch_get_stats(b, out);
}

}  // extern "C"

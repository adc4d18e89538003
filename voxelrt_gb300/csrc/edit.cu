// edit.cu - the edit path on the device: sphere fill/carve on device bricks, brick
// allocation for fills and empty-brick GC, with the occupancy and voxel codes of every
// edited brick re-derived in the same kernel, and no host round trip.
//
// Semantics of VoxelMap::RegionDispatchSIMD + GC (src/VoxelRT/VoxelMap.h:222-263)
// driving the brush (src/VoxelRT/Brush.cpp:10-31), per edit in order: every brick in the
// edit's brick bounding box is visited (created first for fills), voxels with
// |v - c|^2 <= r^2 are set, and visited bricks that end up empty are freed.  Because
// voxels are independent, a batch of edits is applied as
//   host (geometry only, no device state): the sectors the edits' boxes touch, per
//       sector the bricks inside a box (`visit`) and the bricks a fill sphere reaches
//       (`create`), and the sector groups whose brick-table entries follow them;
//   1. edit_sectors_kernel: a cluster of blocks per touched sector, a warp per brick: applies
//      every edit of the batch in order to the visited bricks, drops the emptied ones, moves the
//      sector to a fresh range from the device's bump allocator (alloc.cu) when it gained
//      bricks or packs it in place when it lost some, and derives the cell masks and voxel
//      codes of what it writes;
//   2. the group masks and brick-table entries of the touched groups (world.cu).
// The final state equals applying the edits one by one.  The call only enqueues this
// work on the stream (one upload of the batch from pinned memory and two kernels); the
// host reads nothing back, except when its bound of the bump pointer says the pool may
// be full, and then it compacts the pool first (alloc.cu).

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <unordered_map>
#include <utility>
#include <vector>

#include "brick_codes.cuh"
#include "edit_geometry.h"
#include "world.h"

namespace vrt {
namespace {

struct alignas(16) EditDev {
    int32_t cx, cy, cz;
    int32_t r2;
    int32_t lo[3], hi[3];  // brick bounding box (inclusive)
    uint32_t material;
    uint32_t replace;
};

// A sector an edit batch touches: bricks inside an edit's box, bricks a fill creates.
struct EditSector {
    unsigned long long visit, create;
    uint32_t sector, pad;
};
static_assert(sizeof(EditSector) == 24, "edit sector records are 24 bytes");

constexpr uint32_t kNoSlot = 0xFFFFFFFFu;

// A cluster of 8 blocks per touched sector, a warp for each of its up to 64 bricks (k-th set
// bit of old | create).  Every brick is read before any is written, so a sector that loses
// bricks is packed in place.  A sector that gains some takes popcount(final mask) slots at the
// bump pointer and leaves its old range as garbage.
// Bound by latency: a stroke touches some twenty sectors, and a brick is a load, a few dozen
// instructions per edit that reaches it and a store.  In one kernel the bricks stay in
// registers between the edits and the layout; as three (grow, edit, shrink, the layouts one
// brick after another with a barrier each) a stroke of 24 spheres of radius 14 took 23 + 9 + 13 us,
// and with the frame after it 107 us, now 50.  8 blocks of 8 warps: 200 spheres of radius 30 over
// the same sectors 520 us, 4 of 16 557 us, 2 of 32 594 us.
// A batch over a whole world is bound by the blocks a SM holds: its warps wait for their
// cluster's barriers.  One sphere of radius 400 over 2,048 full sectors, the kernel alone: 132 us with
// every thread reading the emptied bits of the 8 blocks, 126 with 16 threads doing so for their
// block, 114 with 8 blocks a SM (32 registers; 6 with the compiler's 40).  1,000 spheres of radius 4:
// 209, 198 and 180 us a call; 200 of radius 30: 140, 140 and 143 us.
constexpr uint32_t kEditWarps = 8, kEditCluster = 8;
__global__ void __cluster_dims__(kEditCluster, 1, 1) __launch_bounds__(kEditWarps * 32, 8)
    edit_sectors_kernel(const EditSector* __restrict__ ts, const EditDev* __restrict__ edits, uint32_t n_edits,
                        SectorRec* __restrict__ sectors, uint32_t sx, uint32_t sz, DevAlloc* __restrict__ alloc,
                        uint8_t* __restrict__ payload, uint4* __restrict__ codes, uint64_t* __restrict__ cell_masks) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ __align__(16) uint8_t sb[kEditWarps][512];
    __shared__ uint32_t s_emptied[2], s_all[2 * kEditCluster], s_base;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, rank = cluster.block_rank();
    const EditSector es = ts[blockIdx.x / kEditCluster];
    const uint32_t s = es.sector;
    const SectorRec rec = sectors[s];
    const uint64_t old = (uint64_t)rec.mask_hi << 32 | rec.mask_lo, nm = old | es.create;
    if (!(nm & es.visit)) return;  // the whole cluster
    if (threadIdx.x < 2) s_emptied[threadIdx.x] = 0;
    __syncthreads();
    // this warp's brick
    const uint32_t k = rank * kEditWarps + wib;
    const bool mine = k < (uint32_t)__popcll(nm);
    const uint32_t b = mine ? warp_nth_bit(nm, k, lane) : 0u;
    const uint64_t bit = 1ull << b;
    const bool had = mine && (old & bit), visited = mine && (es.visit & bit);
    const uint32_t src = rec.base + (uint32_t)__popcll(old & (bit - 1));
    uint4 v = make_uint4(0, 0, 0, 0);
    if (visited) {
        if (had) v = reinterpret_cast<const uint4*>(payload + (size_t)src * 512)[lane];
        const int32_t bx = (int32_t)((s % sx) * 4 + (b & 3u)), bz = (int32_t)(((s / sx) % sz) * 4 + ((b >> 2) & 3u)),
                      by = (int32_t)((s / (sx * sz)) * 4 + (b >> 4));
        uint8_t* bytes = reinterpret_cast<uint8_t*>(&v);
        // lane holds voxels 16*lane .. 16*lane+15: y = lane>>2, z = 2*(lane&3) + (j>>3), x = j&7
        const int32_t y = by * 8 + (int32_t)(lane >> 2), z0 = bz * 8 + 2 * (int32_t)(lane & 3), x0 = bx * 8;
        for (uint32_t e0 = 0; e0 < n_edits; e0 += 32) {
            // 32 edits at a time: each lane tests one against the brick
            EditDev ed{};
            const bool valid = e0 + lane < n_edits;
            if (valid) ed = edits[e0 + lane];
            uint32_t todo = __ballot_sync(0xffffffffu, valid && bx >= ed.lo[0] && bx <= ed.hi[0] && by >= ed.lo[1] &&
                                                           by <= ed.hi[1] && bz >= ed.lo[2] && bz <= ed.hi[2]);
            for (; todo; todo &= todo - 1) {
                const int l = __ffs(todo) - 1;
                const int32_t dy = y - __shfl_sync(0xffffffffu, ed.cy, l), dz0 = z0 - __shfl_sync(0xffffffffu, ed.cz, l),
                              dx0 = x0 - __shfl_sync(0xffffffffu, ed.cx, l);
                const int32_t r2 = __shfl_sync(0xffffffffu, ed.r2, l);
                const uint32_t paint = __shfl_sync(0xffffffffu, ed.material | ed.replace << 8, l);
                const int32_t left[2] = {r2 - dy * dy - dz0 * dz0, r2 - dy * dy - (dz0 + 1) * (dz0 + 1)};
                const bool replace = paint >> 8 != 0;
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int32_t dx = dx0 + (j & 7);
                    if (dx * dx > left[j >> 3]) continue;
                    if (replace && bytes[j] == 0) continue;
                    bytes[j] = (uint8_t)paint;
                }
            }
        }
        if (!__any_sync(0xffffffffu, (v.x | v.y | v.z | v.w) != 0) && lane == 0)
            atomicOr(&s_emptied[b >> 5], 1u << (b & 31));
    }
    cluster.sync();
    if (threadIdx.x < 2 * kEditCluster)
        s_all[threadIdx.x] = cluster.map_shared_rank(s_emptied, threadIdx.x >> 1)[threadIdx.x & 1];
    __syncthreads();
    uint32_t gone[2] = {0, 0};
#pragma unroll
    for (uint32_t r = 0; r < 2 * kEditCluster; r++) gone[r & 1] |= s_all[r];
    const uint64_t emptied = (uint64_t)gone[0] | (uint64_t)gone[1] << 32;
    const uint64_t fm = nm & ~emptied;
    uint32_t base = rec.base;
    if (fm != old) {  // a new layout
        if (rank == 0 && threadIdx.x == 0) {
            const uint32_t n_new = (uint32_t)__popcll(fm), n_old = (uint32_t)__popcll(old);
            if (fm & ~old) {
                base = atomicAdd(&alloc->top, n_new);
                if ((uint64_t)base + n_new > alloc->cap) {
                    atomicExch(&alloc->overflow, 1u);  // never, while the host's bound of the pointer holds
                    base = kNoSlot;
                }
            }
            if (base != kNoSlot) {
                atomicAdd(&alloc->live, n_new - n_old);
                SectorRec out = rec;
                out.mask_lo = (uint32_t)fm;
                out.mask_hi = (uint32_t)(fm >> 32);
                out.base = fm ? base : 0;
                sectors[s] = out;
            }
            s_base = base;
        }
        // bricks no edit visits that change slots: read before anything is written
        if (mine && !visited) v = reinterpret_cast<const uint4*>(payload + (size_t)src * 512)[lane];
        cluster.sync();
        base = *cluster.map_shared_rank(&s_base, 0);
    }
    // no block may leave while another reads its shared memory: said here, waited for at the end
    auto token = cluster.barrier_arrive();
    const uint32_t dst = base + (uint32_t)__popcll(fm & (bit - 1));
    if (mine && (fm & bit) && base != kNoSlot && (visited || dst != src))
        store_brick(sb[wib], v, dst, lane, payload, codes, cell_masks);
    cluster.barrier_wait(std::move(token));
}

size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

}  // namespace
}  // namespace vrt

using namespace vrt;

extern "C" vrt_status vrt_world_edit(vrt_world* w, const vrt_edit* edits, uint32_t n, void* stream_) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK) return st;
    if (n == 0) return VRT_OK;
    if (!edits) {
        set_error("null edit array");
        return VRT_ERR_INVALID_ARG;
    }
    for (uint32_t i = 0; i < n; i++)
        if (edits[i].radius > 4096 || edits[i].mode > VRT_EDIT_REPLACE || edits[i].reserved) {
            set_error("edit radius must be <= 4096, mode FILL or REPLACE, reserved 0");
            return VRT_ERR_INVALID_ARG;
        }
    std::lock_guard<std::mutex> lock(w->mu);
    cudaStream_t stream = (cudaStream_t)stream_;
    // edits of a world follow each other whatever streams they are queued on
    VRT_CUDA(cudaStreamWaitEvent(stream, w->edited, 0));
    const int32_t nb[3] = {(int32_t)w->sx * 4, (int32_t)w->sy * 4, (int32_t)w->sz * 4};
    // host: geometry of the batch
    std::vector<EditDev> ed(n);
    std::unordered_map<uint32_t, uint32_t> index;  // sector -> position in `secs`
    std::vector<EditSector> secs;
    for (uint32_t i = 0; i < n; i++) {
        const vrt_edit& e = edits[i];
        EditDev& d = ed[i];
        d.cx = e.center[0];
        d.cy = e.center[1];
        d.cz = e.center[2];
        d.r2 = (int32_t)(e.radius * e.radius);
        d.material = e.material;
        d.replace = e.mode == VRT_EDIT_REPLACE;
        bool empty_box = false;
        for (int c = 0; c < 3; c++) {
            const int64_t lo = ((int64_t)e.center[c] - e.radius) >> 3, hi = ((int64_t)e.center[c] + e.radius) >> 3;
            d.lo[c] = (int32_t)std::max<int64_t>(lo, 0);
            d.hi[c] = (int32_t)std::min<int64_t>(hi, nb[c] - 1);
            if (d.lo[c] > d.hi[c]) empty_box = true;
        }
        if (empty_box) {
            d.lo[0] = 1, d.hi[0] = 0;  // never matches
            continue;
        }
        const bool creates = e.material != 0 && e.mode == VRT_EDIT_FILL;
        for (int32_t sy = d.lo[1] >> 2; sy <= d.hi[1] >> 2; sy++)
            for (int32_t sz = d.lo[2] >> 2; sz <= d.hi[2] >> 2; sz++)
                for (int32_t sx = d.lo[0] >> 2; sx <= d.hi[0] >> 2; sx++) {
                    int32_t lo[3], hi[3];
                    const int32_t sc[3] = {sx, sy, sz};
                    for (int c = 0; c < 3; c++) {
                        lo[c] = std::max(d.lo[c], sc[c] * 4) - sc[c] * 4;
                        hi[c] = std::min(d.hi[c], sc[c] * 4 + 3) - sc[c] * 4;
                    }
                    const uint32_t s = w->lin(sx, sy, sz);
                    auto it = index.find(s);
                    if (it == index.end()) {
                        it = index.emplace(s, (uint32_t)secs.size()).first;
                        secs.push_back(EditSector{0, 0, s, 0});
                    }
                    EditSector& es = secs[it->second];
                    es.visit |= box_bits(lo, hi);
                    if (!creates) continue;
                    if (sphere_reaches_all(e, sc, lo, hi)) {
                        es.create |= box_bits(lo, hi);
                        continue;
                    }
                    for (int32_t y = lo[1]; y <= hi[1]; y++)
                        for (int32_t z = lo[2]; z <= hi[2]; z++)
                            for (int32_t x = lo[0]; x <= hi[0]; x++)
                                if (sphere_reaches_brick(e, sx * 4 + x, sy * 4 + y, sz * 4 + z))
                                    es.create |= 1ull << (x | z << 2 | y << 4);
                }
    }
    if (secs.empty()) return VRT_OK;
    // sector groups whose brick-table entries follow the touched sectors
    const uint32_t gx = (w->sx + 3) / 4, gz = (w->sz + 3) / 4;
    std::vector<uint32_t> groups;
    groups.reserve(secs.size());
    uint64_t growing = 0;
    for (const EditSector& es : secs) {
        const uint32_t x = es.sector % w->sx, z = (es.sector / w->sx) % w->sz, y = es.sector / (w->sx * w->sz);
        groups.push_back((x >> 2) + (z >> 2) * gx + (y >> 2) * gx * gz);
        growing += es.create ? 1 : 0;
    }
    std::sort(groups.begin(), groups.end());
    groups.erase(std::unique(groups.begin(), groups.end()), groups.end());
    // a growing sector takes at most 64 slots from the bump pointer
    const uint64_t need = growing * 64;
    if ((st = ensure_headroom(w, need, stream)) != VRT_OK) return st;
    // one upload: [edits][touched sectors][groups], from pinned memory; the stages are
    // used in turn, so a call waits on the host only for the upload four edits back
    const uint32_t m = (uint32_t)secs.size();
    const size_t eb = ed.size() * sizeof(EditDev), sb = secs.size() * sizeof(EditSector);
    const size_t soff = align16(eb), goff = align16(soff + sb), total = goff + groups.size() * sizeof(uint32_t);
    HostStage& stage = w->edit_stage[w->edit_stage_next];
    w->edit_stage_next = (w->edit_stage_next + 1) % 4;
    VRT_CUDA(stage.acquire(total));
    uint8_t* h = (uint8_t*)stage.ptr;
    std::memcpy(h, ed.data(), eb);
    std::memcpy(h + soff, secs.data(), sb);
    std::memcpy(h + goff, groups.data(), groups.size() * sizeof(uint32_t));
    VRT_CUDA(w->d_edit.reserve(total, true));
    uint8_t* d = (uint8_t*)w->d_edit.ptr;
    VRT_CUDA(cudaMemcpyAsync(d, h, total, cudaMemcpyHostToDevice, stream));
    VRT_CUDA(stage.release(stream));
    const EditSector* d_secs = (const EditSector*)(d + soff);
    edit_sectors_kernel<<<m * kEditCluster, kEditWarps * 32, 0, stream>>>(
        d_secs, (const EditDev*)d, n, w->d_sectors, w->sx, w->sz, w->d_alloc, w->d_payload, w->d_codes, w->d_cells);
    VRT_CUDA(cudaGetLastError());
    if ((st = rebuild_table_groups(w, (const uint32_t*)(d + goff), (uint32_t)groups.size(), stream)) != VRT_OK)
        return st;
    VRT_CUDA(cudaEventRecord(w->edited, stream));
    w->host_stale = true;
    w->top_bound += need;
    return VRT_OK;
}

// world.cu - device-resident brickmap storage: create/destroy, dirty-brick sync,
// brick-slot repacking, occupancy re-derivation and the brick table.
//
// Replaces GpuVoxelStorage (src/VoxelRT/GpuRenderer.cpp:17-167) and the
// UpdateOccupancy dispatch (GpuRenderer.cpp:163-166, Shaders/UpdateOccupancy.comp).
// Unlike the reference, bricks that keep their content but change slot are moved
// on the device instead of being re-uploaded from the host
// (BrickSlotAllocator.cpp:84-87 marks the whole sector dirty).

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "brick_codes.cuh"
#include "launch_rules.h"
#include "world.h"

namespace vrt {

vrt_status cuda_fail(cudaError_t e, const char* what) {
    set_error(std::string(what) + ": " + cudaGetErrorString(e));
    if (e == cudaErrorMemoryAllocation) return VRT_ERR_OUT_OF_MEMORY;
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return VRT_ERR_NO_DEVICE;
    return VRT_ERR_DEVICE;
}

vrt_status world_enter(vrt_world* world, DeviceScope& scope) {
    if (!world) {
        set_error("null world");
        return VRT_ERR_INVALID_ARG;
    }
    VRT_CUDA(scope.enter(world->device));
    return VRT_OK;
}

uint32_t sm_count() {
    static std::atomic<int> known[64];  // per device, 0 = not asked yet
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    const bool keep = dev >= 0 && dev < 64;
    if (keep) sms = known[dev].load(std::memory_order_relaxed);
    if (sms == 0) {
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 1;
        if (keep) known[dev].store(sms, std::memory_order_relaxed);
    }
    return (uint32_t)sms;
}

vrt_status L2Window::enter(const vrt_world* w, cudaStream_t s) {
    if (!w || !(w->flags & VRT_WORLD_L2_PERSIST) || !s || w->l2_window_bytes == 0) return VRT_OK;
    VRT_CUDA(cudaStreamGetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &prev));
    cudaStreamAttrValue a{};
    a.accessPolicyWindow.base_ptr = w->d_bricks;
    a.accessPolicyWindow.num_bytes = w->l2_window_bytes;
    a.accessPolicyWindow.hitRatio = w->l2_hit_ratio;
    a.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    a.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    VRT_CUDA(cudaStreamSetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &a));
    stream = s;
    set = true;
    return VRT_OK;
}

L2Window::~L2Window() {
    if (set) cudaStreamSetAttribute(stream, cudaStreamAttributeAccessPolicyWindow, &prev);
}

namespace {

// The window of a VRT_WORLD_L2_PERSIST world: its brick table, up to the device's largest
// window, with the context's persisting L2 set-aside raised to cover it (up to the
// device's maximum; the set-aside lasts as long as this process's context).
vrt_status setup_l2_window(vrt_world* w) {
    int max_window = 0, max_persist = 0;
    VRT_CUDA(cudaDeviceGetAttribute(&max_window, cudaDevAttrMaxAccessPolicyWindowSize, w->device));
    VRT_CUDA(cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, w->device));
    if (max_window <= 0 || max_persist <= 0) return VRT_OK;  // no persisting L2: the flag does nothing
    const size_t table = w->num_brick_positions() * sizeof(uint32_t);
    w->l2_window_bytes = std::min(table, (size_t)max_window);
    size_t limit = 0;
    VRT_CUDA(cudaDeviceGetLimit(&limit, cudaLimitPersistingL2CacheSize));
    const size_t want = std::min(w->l2_window_bytes, (size_t)max_persist);
    if (want > limit) VRT_CUDA(cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, want));
    VRT_CUDA(cudaDeviceGetLimit(&limit, cudaLimitPersistingL2CacheSize));
    w->l2_hit_ratio = (float)std::min(1.0, (double)limit / (double)w->l2_window_bytes);
    return VRT_OK;
}

// ---------------------------------------------------------------------------
// Sector sync.

// One sector of a sync batch, in its new layout: bricks whose bytes were supplied, bricks that
// keep their content but change slot (gathered to scratch before anything is written), and new
// bricks without bytes (zero-filled); the other bricks of `mask` stay as they are.
struct alignas(16) SectorOp {
    uint64_t mask, dirty, moved, fresh;
    uint32_t sector, base;   // 0-based slot of the first brick
    uint32_t first_dirty;    // staged brick of the lowest dirty bit
    uint32_t first_moved;    // scratch brick of the lowest moved bit
};
static_assert(sizeof(SectorOp) == 48, "sector ops are read as three 16-byte words");

// The device allocator's state after a batch (DevAlloc), written by its sync kernel.
struct AllocState {
    DevAlloc* alloc;
    uint32_t top, live, cap;
};

// Payload of the listed slots to scratch, a warp per brick.
__global__ void __launch_bounds__(256)
    gather_bricks_kernel(const uint32_t* __restrict__ slots, uint32_t n, const uint8_t* __restrict__ payload,
                         uint8_t* __restrict__ scratch) {
    const uint32_t lane = threadIdx.x & 31, k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (k >= n) return;
    reinterpret_cast<uint4*>(scratch + (size_t)k * 512)[lane] =
        reinterpret_cast<const uint4*>(payload + (size_t)slots[k] * 512)[lane];
}

// A block per sector op, each of its 16 warps every 16th brick to write (up to 4, loaded
// before the first is stored): payload, cell masks and voxel codes, then the sector's record.
// Bound by memory: 512 B in and 1088 B out a brick.  One op per sector, read from the
// host's pinned list, where a list of 60,000 brick ops took the host longer to build than the
// copy to upload: 60 k bricks of a 512x256x512 terrain synced and a 640x360 frame: 450 us with
// brick ops, 272 us.
constexpr uint32_t kSyncWarps = 16;
__global__ void __launch_bounds__(kSyncWarps * 32)
    sync_sectors_kernel(const SectorOp* __restrict__ ops, const uint8_t* __restrict__ stage,
                        const uint8_t* __restrict__ scratch, AllocState state, SectorRec* __restrict__ sectors,
                        uint8_t* __restrict__ payload, uint4* __restrict__ codes, uint64_t* __restrict__ cells) {
    __shared__ __align__(16) uint8_t sb[kSyncWarps][512];
    __shared__ SectorOp op;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (threadIdx.x < 3)
        reinterpret_cast<uint4*>(&op)[threadIdx.x] = reinterpret_cast<const uint4*>(ops + blockIdx.x)[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
        sectors[op.sector] = SectorRec{(uint32_t)op.mask, (uint32_t)(op.mask >> 32), op.base, 0};
        if (blockIdx.x == 0) {
            state.alloc->top = state.top;
            state.alloc->live = state.live;
            state.alloc->cap = state.cap;
        }
    }
    const uint64_t write = op.dirty | op.moved | op.fresh;
    const uint32_t n = (uint32_t)__popcll(write);
    uint4 v[4];
    uint32_t dst[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        const uint32_t k = wib + j * kSyncWarps;
        if (k >= n) break;
        const uint32_t b = warp_nth_bit(write, k, lane);
        const uint64_t bit = 1ull << b;
        dst[j] = op.base + (uint32_t)__popcll(op.mask & (bit - 1));
        v[j] = make_uint4(0, 0, 0, 0);
        if (op.dirty & bit)
            v[j] = __ldcs(reinterpret_cast<const uint4*>(
                              stage + (size_t)(op.first_dirty + (uint32_t)__popcll(op.dirty & (bit - 1))) * 512) + lane);
        else if (op.moved & bit)
            v[j] = __ldcs(reinterpret_cast<const uint4*>(
                              scratch + (size_t)(op.first_moved + (uint32_t)__popcll(op.moved & (bit - 1))) * 512) + lane);
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        if (wib + j * kSyncWarps >= n) break;
        store_brick(sb[wib], v[j], dst[j], lane, payload, codes, cells);
        __syncwarp();
    }
}

// The brick-table entry of brick b of sector s, written at its brick position; group_mask: the
// mask of the sector's group.
__device__ __forceinline__ void write_table_entry(const SectorRec* __restrict__ sectors,
                                                  const unsigned long long* group_mask, uint32_t s, uint32_t b,
                                                  uint32_t sx, uint32_t sz, uint32_t* __restrict__ bricks) {
    const SectorRec rec = sectors[s];
    const uint32_t x = s % sx, z = (s / sx) % sz, y = s / (sx * sz);
    const uint32_t bx = x * 4 + (b & 3), bz = z * 4 + ((b >> 2) & 3), by = y * 4 + (b >> 4);
    const uint32_t lo = rec.mask_lo, hi = rec.mask_hi;
    uint32_t e;
    if ((((b < 32 ? lo : hi) >> (b & 31)) & 1u) != 0) {
        const uint32_t below = (1u << (b & 31)) - 1u;
        e = rec.base + (b < 32 ? __popc(lo & below) : __popc(lo) + __popc(hi & below));
    } else {
        const uint32_t cpu_m = (8u << skip_levels(lo, hi, b)) - 1u;
        e = kBrickEmpty | cpu_m;
        // the level the GLSL mode and its anisotropic LODs read: the sector's mask, or
        // where the sector is empty its group's mask, at the sector's index in the group
        uint64_t lm = (uint64_t)hi << 32 | lo;
        uint32_t li = b;
        if ((lo | hi) == 0) {
            lm = *group_mask;
            li = (x & 3) | (z & 3) << 2 | (y & 3) << 4;
            e |= kAnisoGroupBit | ((32u << skip_levels((uint32_t)lm, (uint32_t)(lm >> 32), li)) - 1u) << 8;
        } else {
            e |= cpu_m << 8;
        }
        // anisotropic LODs: that mask's skip level per ray octant
        for (uint32_t o = 0; o < 8; o++) {
            const uint64_t f = lm & forward_cells(li, (o & 1u) ? 0 : -1, (o & 2u) ? 0 : -1, (o & 4u) ? 0 : -1);
            e |= skip_levels((uint32_t)f, (uint32_t)(f >> 32), li) << (kAnisoShift + 2 * o);
        }
    }
    bricks[bx + bz * (sx * 4) + by * (sx * 4) * (sz * 4)] = e;
}

// Masks of sector groups, the GLSL mode's 4th level (VoxelTraversal.glsl:114-118): per group of
// 4^3 sectors (index x + z*GX + y*GX*GZ) bit x | z<<2 | y<<4 set when that sector holds a brick
// (GpuRenderer.cpp:139-149); and the brick-table entries of the groups' sectors, 16 blocks of
// 256 threads per group of the list, or of every group without one.  After an edit, only the
// groups of the sectors it changed are re-derived (a sector's emptiness changes its group's
// mask, which the GLSL entries of the group's empty sectors read).  Each block derives the
// mask from the 64 sector records itself, so no pass over all groups goes before (1.4 us and
// a gap of 3 us between the kernels).
__global__ void __launch_bounds__(256)
    brick_table_groups_kernel(const SectorRec* __restrict__ sectors, unsigned long long* __restrict__ groups,
                              const uint32_t* __restrict__ list, uint32_t sx, uint32_t sy, uint32_t sz,
                              uint32_t* __restrict__ bricks) {
    __shared__ uint32_t s_half[2];
    __shared__ unsigned long long s_mask;
    const uint32_t g = list ? list[blockIdx.x >> 4] : blockIdx.x >> 4, gx = (sx + 3) / 4, gz = (sz + 3) / 4;
    const uint32_t x0 = (g % gx) * 4, z0 = ((g / gx) % gz) * 4, y0 = (g / (gx * gz)) * 4;
    if (threadIdx.x < 64) {
        const uint32_t b = threadIdx.x, x = x0 + (b & 3u), z = z0 + ((b >> 2) & 3u), y = y0 + (b >> 4);
        bool nonempty = false;
        if (x < sx && y < sy && z < sz) {
            const SectorRec r = sectors[x + z * sx + y * sx * sz];
            nonempty = (r.mask_lo | r.mask_hi) != 0;
        }
        const uint32_t half = __ballot_sync(0xffffffffu, nonempty);
        if ((b & 31u) == 0) s_half[b >> 5] = half;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_mask = (unsigned long long)s_half[0] | (unsigned long long)s_half[1] << 32;
        if ((blockIdx.x & 15u) == 0) groups[g] = s_mask;
    }
    __syncthreads();
    const uint32_t i = (blockIdx.x & 15u) * 256 + threadIdx.x, si = i >> 6;
    const uint32_t x = x0 + (si & 3u), z = z0 + ((si >> 2) & 3u), y = y0 + (si >> 4);
    if (x >= sx || y >= sy || z >= sz) return;
    write_table_entry(sectors, &s_mask, x + z * sx + y * sx * sz, i & 63u, sx, sz, bricks);
}

// ---------------------------------------------------------------------------

// Grow the brick pools to at least min_capacity slots (at least doubling);
// slots keep their content, so planned moves stay valid.
vrt_status grow_pool(vrt_world* w, uint32_t min_capacity, cudaStream_t stream) {
    uint64_t want = std::max<uint64_t>({(uint64_t)w->capacity * 2, (uint64_t)min_capacity, 1024});
    want = std::min<uint64_t>(want, 0x3fffffffull);
    if (want <= w->capacity) {
        set_error("brick pool cannot grow further");
        return VRT_ERR_SLOTS_EXHAUSTED;
    }
    uint32_t cap = (uint32_t)want;
    uint4* codes = nullptr;
    uint8_t* payload = nullptr;
    uint64_t* cells = nullptr;
    cudaError_t e = cudaMalloc(&codes, (size_t)cap * 512);
    if (e == cudaSuccess) e = cudaMalloc(&payload, (size_t)cap * 512);
    if (e == cudaSuccess) e = cudaMalloc(&cells, (size_t)cap * 64);
    if (e != cudaSuccess) {
        if (codes) cudaFree(codes);
        if (payload) cudaFree(payload);
        cudaGetLastError();
        return cuda_fail(e, "grow brick pool");
    }
    if (w->capacity) {
        VRT_CUDA(cudaMemcpyAsync(codes, w->d_codes, (size_t)w->capacity * 512, cudaMemcpyDeviceToDevice, stream));
        VRT_CUDA(cudaMemcpyAsync(payload, w->d_payload, (size_t)w->capacity * 512, cudaMemcpyDeviceToDevice, stream));
        VRT_CUDA(cudaMemcpyAsync(cells, w->d_cells, (size_t)w->capacity * 64, cudaMemcpyDeviceToDevice, stream));
        VRT_CUDA(cudaStreamSynchronize(stream));
    }
    if (w->d_codes) cudaFree(w->d_codes);
    if (w->d_payload) cudaFree(w->d_payload);
    if (w->d_cells) cudaFree(w->d_cells);
    w->d_codes = codes;
    w->d_payload = payload;
    w->d_cells = cells;
    w->capacity = cap;
    w->arena.grow(cap);
    return VRT_OK;
}

// One self-consistent batch of sector updates: plan, then gather, then write.
struct SyncBatch {
    std::vector<SectorOp> ops;
    std::vector<uint32_t> gathers;   // old slots of moved bricks, copied to scratch first
    const uint8_t* src = nullptr;    // first input brick of the batch
    uint64_t n_stage = 0;            // bricks staged from the input
};

vrt_status plan_sector(vrt_world* w, SyncBatch& b, uint32_t s, uint64_t am, uint64_t dm, uint64_t stage_first,
                       cudaStream_t stream) {
    SectorSlots& cur = w->slots[s];
    const SectorSlots old = cur;
    sector_free(w->arena, cur, old.mask & ~am);
    while (!sector_alloc(w->arena, cur, am)) {
        vrt_status st = grow_pool(w, w->capacity + 64, stream);
        if (st != VRT_OK) return st;
    }
    SectorOp op{};
    op.mask = cur.mask;
    op.dirty = dm & cur.mask;
    op.fresh = cur.mask & ~op.dirty & ~old.mask;
    op.sector = s;
    op.base = cur.base ? cur.base - 1 : 0;
    op.first_dirty = (uint32_t)stage_first;
    op.first_moved = (uint32_t)b.gathers.size();
    for (uint64_t r = cur.mask & ~op.dirty & old.mask; r; r &= r - 1) {
        const uint32_t brick = (uint32_t)__builtin_ctzll(r), src = old.slot_of(brick) - 1;
        if (src == cur.slot_of(brick) - 1) continue;
        op.moved |= 1ull << brick;
        b.gathers.push_back(src);
    }
    b.ops.push_back(op);
    w->h_table[s] = SectorRec{(uint32_t)cur.mask, (uint32_t)(cur.mask >> 32), op.base, 0};
    return VRT_OK;
}

}  // namespace

vrt_status rebuild_table_groups(vrt_world* w, const uint32_t* groups, uint32_t n, cudaStream_t stream) {
    if (groups && n == 0) return VRT_OK;
    const bool all = !groups || (uint64_t)n * 4 >= w->num_groups();
    brick_table_groups_kernel<<<(all ? w->num_groups() : n) * 16u, 256, 0, stream>>>(
        w->d_sectors, (unsigned long long*)w->d_groups, all ? nullptr : groups, w->sx, w->sy, w->sz, w->d_bricks);
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

namespace {

size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

vrt_status run_batch(vrt_world* w, SyncBatch& b, cudaStream_t stream) {
    if (b.ops.empty()) return VRT_OK;
    const size_t stage_bytes = (size_t)b.n_stage * 512;
    if (stage_bytes) {
        VRT_CUDA(w->d_stage.reserve(stage_bytes));
        VRT_CUDA(cudaMemcpyAsync(w->d_stage.ptr, b.src, stage_bytes, cudaMemcpyHostToDevice, stream));
    }
    // sector groups whose brick-table entries follow the sectors
    const uint32_t gx = (w->sx + 3) / 4, gz = (w->sz + 3) / 4;
    std::vector<uint32_t> groups;
    groups.reserve(b.ops.size());
    for (const SectorOp& op : b.ops) {
        const uint32_t x = op.sector % w->sx, z = (op.sector / w->sx) % w->sz, y = op.sector / (w->sx * w->sz);
        groups.push_back((x >> 2) + (z >> 2) * gx + (y >> 2) * gx * gz);
    }
    std::sort(groups.begin(), groups.end());
    groups.erase(std::unique(groups.begin(), groups.end()), groups.end());
    // the kernels read the lists where they are, in pinned memory (a few bytes per sector)
    const size_t ng = b.gathers.size(), ob = b.ops.size() * sizeof(SectorOp);
    const size_t goff = align16(ob), loff = align16(goff + ng * sizeof(uint32_t));
    VRT_CUDA(w->sync_stage.acquire(loff + groups.size() * sizeof(uint32_t)));
    uint8_t* h = (uint8_t*)w->sync_stage.ptr;
    std::memcpy(h, b.ops.data(), ob);
    if (ng) std::memcpy(h + goff, b.gathers.data(), ng * sizeof(uint32_t));
    std::memcpy(h + loff, groups.data(), groups.size() * sizeof(uint32_t));
    if (ng) {
        VRT_CUDA(w->d_scratch.reserve(ng * 512, true));
        gather_bricks_kernel<<<(uint32_t)((ng + 7) / 8), 256, 0, stream>>>((const uint32_t*)(h + goff), (uint32_t)ng,
                                                                          w->d_payload, (uint8_t*)w->d_scratch.ptr);
        VRT_CUDA(cudaGetLastError());
    }
    w->top_bound = w->arena.high_water() - 1;  // as alloc_publish
    const AllocState state{w->d_alloc, (uint32_t)w->top_bound, w->arena.allocated(), w->capacity};
    sync_sectors_kernel<<<(uint32_t)b.ops.size(), kSyncWarps * 32, 0, stream>>>(
        (const SectorOp*)h, (const uint8_t*)w->d_stage.ptr, (const uint8_t*)w->d_scratch.ptr, state, w->d_sectors,
        w->d_payload, w->d_codes, w->d_cells);
    VRT_CUDA(cudaGetLastError());
    vrt_status st = rebuild_table_groups(w, (const uint32_t*)(h + loff), (uint32_t)groups.size(), stream);
    if (st != VRT_OK) return st;
    VRT_CUDA(cudaStreamSynchronize(stream));
    b.ops.clear();
    b.gathers.clear();
    b.n_stage = 0;
    return VRT_OK;
}

}  // namespace

}  // namespace vrt

using namespace vrt;

extern "C" {

const char* vrt_last_error(void) { return vrt::last_error_cstr(); }

uint32_t vrt_abi_version(void) { return VRT_ABI_VERSION; }

int32_t vrt_sector_index(int32_t sx, int32_t sy, int32_t sz) { return sector_index_pack(sx, sy, sz); }

vrt_status vrt_world_create(const vrt_world_desc* desc, vrt_world** out) {
    if (!desc || !out) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    *out = nullptr;
    if (desc->sectors_x == 0 || desc->sectors_y == 0 || desc->sectors_z == 0 ||
        desc->sectors_x * 32 > VRT_MAX_WORLD_X || desc->sectors_y * 32 > VRT_MAX_WORLD_Y ||
        desc->sectors_z * 32 > VRT_MAX_WORLD_Z) {
        set_error("world extent must be 1..64 x 1..32 x 1..64 sectors");
        return VRT_ERR_INVALID_ARG;
    }
    if (desc->flags & ~VRT_WORLD_L2_PERSIST) {
        set_error("unknown world flags");
        return VRT_ERR_INVALID_ARG;
    }
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error("no CUDA device");
        return VRT_ERR_NO_DEVICE;
    }
    if (desc->device < 0 || desc->device >= ndev) {
        set_error("device ordinal out of range");
        return VRT_ERR_INVALID_ARG;
    }
    vrt_world* w = new vrt_world;
    w->device = desc->device;
    w->sx = desc->sectors_x;
    w->sy = desc->sectors_y;
    w->sz = desc->sectors_z;
    w->flags = desc->flags;
    w->slots.assign(w->num_sectors(), SectorSlots{});
    w->h_table.assign(w->num_sectors(), SectorRec{0, 0, 0, 0});
    w->sync_mark.assign(w->num_sectors(), 0);
    w->arena.reset(0);
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st == VRT_OK) {
        e = cudaMalloc(&w->d_sectors, (size_t)w->num_sectors() * sizeof(SectorRec));
        if (e == cudaSuccess) e = cudaMemset(w->d_sectors, 0, (size_t)w->num_sectors() * sizeof(SectorRec));
        if (e == cudaSuccess) e = cudaMalloc(&w->d_bricks, w->num_brick_positions() * sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMalloc(&w->d_groups, (size_t)w->num_groups() * sizeof(uint64_t));
        if (e == cudaSuccess) e = cudaMalloc(&w->d_alloc, sizeof(DevAlloc));
        if (e == cudaSuccess) e = cudaMemset(w->d_alloc, 0, sizeof(DevAlloc));
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&w->edited, cudaEventDisableTiming);
        // edit scratch for batches of up to a few thousand touched sectors: a buffer that
        // grows later frees its old block, and cudaFree waits for the whole device
        if (e == cudaSuccess) e = w->d_edit.reserve(256 << 10);
        for (auto& stage : w->edit_stage)
            if (e == cudaSuccess) e = stage.acquire(64 << 10);
        if (e == cudaSuccess) e = w->sync_stage.acquire(64 << 10);
        if (e != cudaSuccess) st = cuda_fail(e, "allocate sector table");
        if (st == VRT_OK) st = rebuild_table_groups(w, nullptr, 0, 0);
        if (st == VRT_OK && (e = cudaStreamSynchronize(0)) != cudaSuccess) st = cuda_fail(e, "build brick table");
    }
    if (st == VRT_OK) st = grow_pool(w, desc->brick_capacity ? desc->brick_capacity : 4096, 0);
    if (st == VRT_OK) st = alloc_publish(w, 0);
    if (st == VRT_OK && (w->flags & VRT_WORLD_L2_PERSIST)) st = setup_l2_window(w);
    if (st == VRT_OK && cudaStreamSynchronize(0) != cudaSuccess) st = cuda_fail(cudaGetLastError(), "create world");
    if (st != VRT_OK) {
        vrt_world_destroy(w);
        return st;
    }
    *out = w;
    return VRT_OK;
}

vrt_status vrt_world_destroy(vrt_world* w) {
    if (!w) return VRT_OK;
    DeviceScope ds;
    ds.enter(w->device);
    cudaDeviceSynchronize();
    if (w->d_sectors) cudaFree(w->d_sectors);
    if (w->d_bricks) cudaFree(w->d_bricks);
    if (w->d_groups) cudaFree(w->d_groups);
    if (w->d_codes) cudaFree(w->d_codes);
    if (w->d_payload) cudaFree(w->d_payload);
    if (w->d_cells) cudaFree(w->d_cells);
    w->d_stage.release();
    w->d_scratch.release();
    w->d_io.release();
    w->sync_stage.destroy();
    w->d_edit.release();
    for (auto& stage : w->edit_stage) stage.destroy();
    if (w->d_alloc) cudaFree(w->d_alloc);
    if (w->edited) cudaEventDestroy(w->edited);
    delete w;
    return VRT_OK;
}

vrt_status vrt_world_get_stats(const vrt_world* cw, vrt_world_stats* out) {
    if (!cw || !out) {
        set_error("null argument");
        return VRT_ERR_INVALID_ARG;
    }
    // the host mirror is rebuilt from the device after device edits (a cache of the
    // device's state, not a change to the world)
    vrt_world* w = const_cast<vrt_world*>(cw);
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK) return st;
    std::lock_guard<std::mutex> lock(w->mu);
    if ((st = refresh_host_mirror(w)) != VRT_OK) return st;
    out->sectors_x = w->sx;
    out->sectors_y = w->sy;
    out->sectors_z = w->sz;
    out->allocated_bricks = w->arena.allocated();
    out->brick_capacity = w->capacity;
    out->free_ranges = (uint32_t)w->arena.num_ranges();
    out->compactions = w->compactions;
    out->reserved = 0;
    // sector records, brick table, group masks, per slot 512 B payload + 512 B codes +
    // 64 B cell masks, and the scratch buffers
    out->device_bytes = (uint64_t)w->num_sectors() * sizeof(SectorRec) + (uint64_t)w->num_brick_positions() * 4 +
                        (uint64_t)w->num_groups() * 8 + (uint64_t)w->capacity * 1088 + w->d_stage.bytes +
                        w->d_scratch.bytes + w->d_io.bytes + w->d_edit.bytes;
    return VRT_OK;
}

vrt_status vrt_world_sync_sectors(vrt_world* w, uint32_t n, const int32_t* sector_idx, const uint64_t* alloc_mask,
                                  const uint64_t* dirty_mask, const uint8_t* bricks, void* stream_) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK) return st;
    if (n && (!sector_idx || !alloc_mask)) {
        set_error("null sector arrays");
        return VRT_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(w->mu);
    if ((st = refresh_host_mirror(w)) != VRT_OK) return st;
    cudaStream_t stream = (cudaStream_t)stream_;
    const uint64_t kBatchBricks = 1ull << 19;  // 256 MiB of staged bricks per batch
    SyncBatch batch;
    batch.ops.reserve(std::min<uint32_t>(n, 1u << 16));
    w->next_sync_batch();
    uint64_t in_brick = 0;  // index of the next brick in the input stream
    for (uint32_t i = 0; i < n; i++) {
        const uint64_t am = alloc_mask[i];
        const uint64_t dm = dirty_mask ? (dirty_mask[i] & am) : am;
        const uint64_t cnt = (uint64_t)__builtin_popcountll(dm);
        if (cnt && !bricks) {
            set_error("null brick data");
            return VRT_ERR_INVALID_ARG;
        }
        int32_t x, y, z;
        sector_index_unpack(sector_idx[i], x, y, z);
        if (w->sector_in(x, y, z)) {
            const uint32_t s = w->lin(x, y, z);
            if (w->sync_mark[s] == w->sync_batch || batch.n_stage + cnt > kBatchBricks) {
                if ((st = run_batch(w, batch, stream)) != VRT_OK) return st;
                w->next_sync_batch();
            }
            if (batch.ops.empty()) {
                batch.src = bricks ? bricks + in_brick * 512 : nullptr;
                batch.n_stage = 0;
            }
            // stage index relative to the batch's first input brick
            const uint64_t first = (bricks ? (in_brick - (uint64_t)(batch.src - bricks) / 512) : 0);
            if ((st = plan_sector(w, batch, s, am, dm, first, stream)) != VRT_OK) return st;
            batch.n_stage = first + cnt;
            w->sync_mark[s] = w->sync_batch;
        }
        in_brick += cnt;
    }
    return run_batch(w, batch, stream);
}

vrt_status vrt_world_save_cvox(vrt_world* w, const char* path) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK) return st;
    std::vector<int32_t> idx;
    std::vector<uint64_t> masks;
    std::vector<uint8_t> bricks;
    {
        std::lock_guard<std::mutex> lock(w->mu);
        if ((st = refresh_host_mirror(w)) != VRT_OK) return st;
        for (uint32_t y = 0; y < w->sy; y++)
            for (uint32_t z = 0; z < w->sz; z++)
                for (uint32_t x = 0; x < w->sx; x++) {
                    const SectorSlots& s = w->slots[w->lin((int32_t)x, (int32_t)y, (int32_t)z)];
                    if (!s.mask) continue;
                    idx.push_back(sector_index_pack((int32_t)x, (int32_t)y, (int32_t)z));
                    masks.push_back(s.mask);
                    const size_t nb = (size_t)__builtin_popcountll(s.mask);
                    const size_t off = bricks.size();
                    bricks.resize(off + nb * 512);
                    VRT_CUDA(cudaMemcpy(bricks.data() + off, w->d_payload + (size_t)(s.base - 1) * 512, nb * 512,
                                        cudaMemcpyDeviceToHost));
                }
    }
    return vrt_cvox_write(path, (uint32_t)idx.size(), idx.data(), masks.data(), bricks.data());
}

vrt_status vrt_world_load_cvox(vrt_world* w, const char* path, void* stream) {
    vrt_sector_stream* s = nullptr;
    vrt_status st = vrt_cvox_read(path, &s);
    if (st != VRT_OK) return st;
    st = vrt_world_sync_sectors(w, s->n_sectors, s->sector_idx, s->alloc_mask, nullptr, s->bricks, stream);
    vrt_sector_stream_free(s);
    return st;
}

vrt_status vrt_world_read_sector(vrt_world* w, int32_t sector_idx, uint64_t* alloc_mask, uint8_t* bricks,
                                 size_t bricks_capacity, void* stream_) {
    DeviceScope ds;
    vrt_status st = world_enter(w, ds);
    if (st != VRT_OK) return st;
    int32_t x, y, z;
    sector_index_unpack(sector_idx, x, y, z);
    if (!w->sector_in(x, y, z)) {
        set_error("sector outside the world");
        return VRT_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(w->mu);
    if ((st = refresh_host_mirror(w)) != VRT_OK) return st;
    const SectorSlots& s = w->slots[w->lin(x, y, z)];
    if (alloc_mask) *alloc_mask = s.mask;
    const size_t need = (size_t)__builtin_popcountll(s.mask) * 512;
    if (!bricks || need == 0) return VRT_OK;
    if (bricks_capacity < need) {
        set_error("brick buffer too small");
        return VRT_ERR_INVALID_ARG;
    }
    cudaStream_t stream = (cudaStream_t)stream_;
    VRT_CUDA(cudaMemcpyAsync(bricks, w->d_payload + (size_t)(s.base - 1) * 512, need, cudaMemcpyDeviceToHost, stream));
    VRT_CUDA(cudaStreamSynchronize(stream));
    return VRT_OK;
}

}  // extern "C"

// queue_sched.cuh -- the tile shapes of the persistent sweeps (sweep_queue.cu: row
// layouts; sweep_split.cu: direction-split layouts) and the row layouts' queue (the
// split sweep's is described and kept in its file).
//
// The grid is the resident capacity of the GPU.  Each CTA takes the next
// (sector, tile) item from a global counter in sector-major order, re-stages
// its step tables only when the sector or the DEM changes, and keeps every
// point's sectors in order: item (s, T) waits, after its sweep and before its
// surface writes, until tile T's counter of completed sectors reaches s.  The
// wait is bounded (TVS_ERR_TIMEOUT in the error word, the item's writes
// skipped, later waits give up at once).
#pragma once

#include <cstdint>

#include "tvs.h"
#include "tvs_internal.cuh"

namespace tvs {

constexpr int kQueueTileX = 32;
// warps per CTA of the persistent sweeps (one build-wide value: the host tiles
// the grid with it)
#ifndef TVS_QUEUE_WARPS
#define TVS_QUEUE_WARPS 8
#endif
constexpr int kQueueTileY = TVS_QUEUE_WARPS;
constexpr int kQueueThreads = kQueueTileX * kQueueTileY;

// Warps per CTA of the split sweep and warp tiles per chunk of its queue.  A CTA
// takes kSplitGrab chunks at a time while many are left: with one tile per warp in
// a slot, a warp whose tiles are skipped for the most part waits for the slowest to
// leave one (3601^2 exact f32 86.2 against 82.9 ms); with 64 tiles to the end the
// CTAs finish unevenly (1201^2 3.71 against 3.88 ms).
constexpr int kSplitWarps = 16;
constexpr uint32_t kSplitChunk = 8, kSplitGrab = 8;

// The split sweep's launches take as many sectors as have planes of surfaces (one
// per sector and direction) of kPlaneBytes, and kPlaneSectors of a large DEM's up
// to kPlaneBytesMost: the end of a launch leaves the GPU half idle for one tile's
// time (12 tiles of up to 1601^2: 65.0, 57.5, 53.6 and 51.8 ms with 32, 64, 128 and
// 256 MB; 3601^2 MIXED64, 23 MB a sector: 103.5, 100.6 and 98.9 ms with 16, 32 and 64
// sectors, exact f32 83.5, 82.4 and 81.3; 7201^2 MIXED64 with 1, 2 and 4 GB: 785, 779
// and 774 ms).
constexpr size_t kPlaneBytes = (size_t)256 << 20, kPlaneBytesMost = (size_t)1 << 30;
constexpr uint32_t kPlaneSectors = 32;

// Direction-split layouts 1-9: a warp holds LX columns x 32/LX rows of lanes;
// each lane sweeps four points of view, LX columns apart (layouts 1-3: LX = 8,
// 16, 32), 2 x 2 of them, LX columns and 32/LX rows apart (layouts 4-6), or
// four rows 32/LX apart in one column (layouts 7, 8: LX = 32, 16), so that one
// load of the warp reads whole 128- or 64-byte rows.  Layout 9 (quad) is layout
// 8's 16 x 8 tile, a lane's four rows consecutive and read as one float4 from the
// DEM's row-interleaved copies: a warp's load is two runs of 256 bytes.  (Against
// a 32 x 4 tile the runs of one step meet the next one's again: 8.1 in place of
// 12.3 new sectors a step, and a small grid wastes fewer lanes at its edges; 1201^2
// exact f32 3.95 -> 3.72 ms.)  The tile of the split sweep's queue is one warp's
// 128 points of view.
constexpr int kSplitCols = 4;  // points of view per lane
constexpr int kSplitLayouts = 9;
__host__ __device__ constexpr int split_lx(int layout) {
    return layout == 7 ? 32 : layout >= 8 ? 16 : 4 << ((layout - 1) % 3 + 1);
}
__host__ __device__ constexpr int split_ky(int layout) { return layout > 6 ? 4 : layout > 3 ? 2 : 1; }
__host__ __device__ constexpr int split_tile_w(int layout) {
    return kSplitCols / split_ky(layout) * split_lx(layout);
}
__host__ __device__ constexpr int split_tile_h(int layout) {
    return 32 / split_lx(layout) * split_ky(layout);
}

struct QueueCtl {
    QueueDem dem;           // the current item's DEM (copied from the descriptor array)
    uint32_t item;
    uint32_t dem_index;     // descriptor index of `dem`
    uint32_t sector;        // the staged sector
    uint32_t tile;          // the current item's tile within its DEM
    int32_t sector_status;  // the staged sector's shape status
    int32_t wait_status;    // this item's dependency wait
    uint32_t n_steps;
    uint32_t n_fast;
    bool restage;
    float hmax;             // the staged DEM's elevation range (estimate windows)
};

#ifdef __CUDACC__
__device__ __forceinline__ void queue_init(QueueCtl &ctl, uint32_t tid) {
    if (tid == 0) {
        ctl.dem_index = 0xFFFFFFFFu;
        ctl.sector = 0xFFFFFFFFu;
    }
}

// Takes the next item (thread 0) and publishes it to the CTA.  Returns false
// (for the whole CTA) when the queue is empty.
__device__ __forceinline__ bool queue_next(const QueueArgs &a, QueueCtl &ctl, uint32_t tid) {
    const uint32_t n_items = a.tiles_per_sector * a.n_sectors;
    if (tid == 0) {
        const uint32_t item = atomicAdd(a.queue, 1u);
        ctl.item = item;
        if (item < n_items) {
            const uint32_t s = item / a.tiles_per_sector;
            const uint32_t r = item - s * a.tiles_per_sector;
            // the DEM whose tiles hold r (tile_base ascends)
            uint32_t lo = 0, hi = a.n_dems - 1;
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1) >> 1;
                if (a.dems[mid].tile_base <= r) lo = mid; else hi = mid - 1;
            }
            ctl.restage = lo != ctl.dem_index || s != ctl.sector;
            if (lo != ctl.dem_index) ctl.dem = a.dems[lo];
            ctl.dem_index = lo;
            ctl.sector = s;
            ctl.tile = r - ctl.dem.tile_base;
        }
    }
    __syncthreads();
    return ctl.item < n_items;
}

// The tile's previous sector must be complete before this sector's surfaces
// are added.  Every thread of the CTA calls it; returns whether to write.
__device__ __forceinline__ bool queue_wait_prev(const QueueArgs &a, QueueCtl &ctl,
                                                const QueueDem &D, uint32_t s, uint32_t tile,
                                                uint32_t tid) {
    if (tid == 0) {
        ctl.wait_status = TVS_OK;
        if (s > 0) {
            const volatile uint32_t *d = a.done + D.done_base + tile;
            const volatile int32_t *err = a.error;
            uint32_t spins = 0;
            while (*d < s) {
                // give up at the limit, or at once when another wait already did
                if (++spins > a.spin_limit || *err != 0) {
                    atomicExch(a.error, (int32_t)TVS_ERR_TIMEOUT);
                    ctl.wait_status = TVS_ERR_TIMEOUT;
                    break;
                }
                __nanosleep(256);
            }
            __threadfence();
        }
    }
    __syncthreads();
    return ctl.wait_status == TVS_OK;
}

// This item's writes are done: advance the tile's counter of completed sectors.
__device__ __forceinline__ void queue_done(const QueueArgs &a, const QueueDem &D, uint32_t tile,
                                           uint32_t tid) {
    __threadfence();  // this thread's surface writes before the tile's counter
    __syncthreads();
    if (tid == 0 && D.done_base + tile != a.held_tile) atomicAdd(a.done + D.done_base + tile, 1u);
}
#endif

// Host: launch of a persistent queue kernel over `items` work items: the
// shared-memory attribute (only ever raised) and the occupancy are kept per
// (kernel, device) under a lock; the queue and tile counters are reset on the
// stream first.
cudaError_t launch_persistent(const void *fn, const QueueArgs &a, uint64_t items, dim3 block,
                              size_t smem, cudaStream_t s, uint32_t n_slots = 0);

}  // namespace tvs

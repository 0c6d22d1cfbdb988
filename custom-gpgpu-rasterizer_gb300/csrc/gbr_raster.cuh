// gbr_raster.cuh -- the raster kernels' work queue.
#pragma once
#include "gbr_device.cuh"

namespace gbr {

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Work item `idx` into shared memory by an asynchronous 16-byte copy (the
// end marker when the queue is drained); cp_async_wait_all() completes it.
__device__ __forceinline__ void fetch_item(uint4* dst, const uint4* items, uint32_t idx, uint32_t num_items) {
    if (idx >= num_items) {
        *dst = make_uint4(0xFFFFFFFFu, 0u, 0u, 0u);
        return;
    }
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(items + idx) : "memory");
}

// The count pass's counters of a frame (Ctl): handed on, and left zero for
// the next frame.
__device__ __forceinline__ void close_counters(Ctl* c) {
    c->num_visible = c->visible;
    c->num_float_path = c->float_path;
    c->visible = c->float_path = c->rank_next = 0u;
}

// A bin that the raster draws in a predicted frame (exact frames: the scan has
// flagged it).  Without a value returned: a byte read, changed and written held
// up the item's first thread (1M soup in the normal view 230 -> 237 us).
__device__ __forceinline__ void mark_drawn(const FrameDev& F, uint32_t bin) {
    if (F.dirty && F.exact_guard) atomicOr(reinterpret_cast<uint32_t*>(F.dirty) + (bin >> 2), kDirtyNow << (8u * (bin & 3u)));
}

// After a fill pass with the scan in it, the raster leaves the bins' counts
// zero for the next frame.
__device__ __forceinline__ void zero_counts(const FrameDev& F) {
    if (F.fused_scan)
        for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < F.count_split * F.num_bins; b += gridDim.x * blockDim.x)
            F.counts[b] = 0u;
}

}  // namespace gbr

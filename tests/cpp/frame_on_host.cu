// frame_on_host.cu -- the host path of a frame (gbr_api.cu) without a GPU: the
// CUDA runtime calls it makes work on host memory (cuda_on_host.cpp), and the
// kernels' launchers are replaced by what they leave behind for the host path -- counts, totals,
// work items, merge words -- from per-bin entry counts that a test sets.  A
// launch can be made to fail, as one does whose code no longer finds room on
// the device.
#include <cstring>
#include <vector>

#include "gbr_device.cuh"
#include "gbr_internal.h"
#include "gbr_kernels.h"
#include "gbr_predict.h"

using namespace gbr;

namespace {
std::vector<uint32_t> g_bins;   // entries of each bin
uint32_t g_visible = 0;
int g_fail = 0;                 // launches until one fails (0: none)
FrameDev g_last;                // the last frame's descriptor

cudaError_t launched() { return g_fail > 0 && --g_fail == 0 ? cudaErrorMemoryAllocation : cudaSuccess; }

// the totals of a scan over the counts that the set-up pass left
void totals(const FrameDev& F) {
    uint64_t pairs = 0, items = 0, base = 0;
    for (uint32_t b = 0; b < F.num_bins; ++b) {
        uint32_t c = 0;
        for (uint32_t k = 0; k < F.count_split; ++k) c += F.counts[k * F.count_stride + b];
        pairs += c;
        items += (c + F.chunk - 1u) / F.chunk;
        base += (c + F.base_chunk - 1u) / F.base_chunk;
    }
    F.ctl->num_pairs = pairs;
    F.ctl->num_items = (uint32_t)items;
    F.ctl->items_alloc = items;
    F.ctl->base_items[0] = (uint32_t)base;
    F.ctl->overflow = pairs > F.list_cap;
}
}  // namespace

extern "C" {
void host_set_bins(const uint32_t* counts, uint32_t n, uint32_t visible) {
    g_bins.assign(counts, counts + n);
    g_visible = visible;
}
void host_fail_launch(int nth) { g_fail = nth; }
void host_last_frame(uint32_t out[4]) {
    out[0] = g_last.chunk;
    out[1] = g_last.block_threads;
    out[2] = g_last.direct;
    out[3] = g_last.fused_scan;
}
}

namespace gbr {
// -- launchers ---------------------------------------------------------
void free_texture(TexHost&) {}
cudaError_t raster_configure(uint32_t, uint32_t, uint32_t, RasterGrid* g) {
    g->block64 = 16; g->block128 = 8; g->block512 = 2; g->record = 6;
    return cudaSuccess;
}
cudaError_t launch_setup(const FrameDev& F, const MeshDev*, bool, cudaStream_t) {
    if (const cudaError_t e = launched()) return e;
    g_last = F;
    F.ctl->visible += g_visible;
    for (uint32_t b = 0; b < F.num_bins; ++b) {
        F.counts[b] += b < g_bins.size() ? g_bins[b] : 0u;
        F.ctl->rank_next += F.row_blocks || b >= g_bins.size() ? 0u : g_bins[b];
    }
    if (F.direct) F.gvis[0] = 7u;   // a triangle drawn by the set-up pass
    return cudaSuccess;
}
ScanDev scan_of(const FrameDev&, uint32_t mode) {
    ScanDev S;
    memset(&S, 0, sizeof S);
    S.mode = mode;
    return S;
}
cudaError_t launch_scan(const ScanDev&, cudaStream_t) {
    if (const cudaError_t e = launched()) return e;
    totals(g_last);
    memset(g_last.counts, 0, (size_t)g_last.count_split * g_last.num_bins * sizeof(uint32_t));
    return cudaSuccess;
}
cudaError_t launch_list_touch(const FrameDev&, cudaStream_t) { return launched(); }
cudaError_t launch_fill(const FrameDev& F, cudaStream_t) {
    if (const cudaError_t e = launched()) return e;
    if (F.fused_scan) totals(F);
    return cudaSuccess;
}
cudaError_t launch_raster(const FrameDev& F, const RasterGrid&, cudaStream_t) {
    if (const cudaError_t e = launched()) return e;
    if (F.fused_scan) memset(F.counts, 0, (size_t)F.count_split * F.num_bins * sizeof(uint32_t));
    F.ctl->num_visible = F.ctl->visible;
    F.ctl->visible = F.ctl->float_path = F.ctl->rank_next = 0u;
    F.gvis[1] = 9u;
    return cudaSuccess;
}
cudaError_t launch_shade(const FrameDev& F, const ShadeOne*, cudaStream_t) {
    if (const cudaError_t e = launched()) return e;
    for (size_t i = 0; i < (size_t)F.width * F.height; ++i) {
        F.ids[i] = (uint32_t)F.gvis[i];
        F.gvis[i] = kEmptyVis;
    }
    return cudaSuccess;
}
cudaError_t launch_prepass(const FrameDev&, cudaStream_t) { return launched(); }
cudaError_t launch_capacity(const FrameDev&, bool, cudaStream_t) { return launched(); }
cudaError_t launch_feat_reset(const FrameDev&, cudaStream_t) { return launched(); }
cudaError_t launch_mlp_predict(const uint16_t*, const float*, uint32_t, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_mlp_grad(const uint16_t*, const float*, const float*, uint32_t, float*, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_mlp_adam(float*, uint16_t*, const float*, float*, float*, uint32_t, float, float, cudaStream_t) { return cudaSuccess; }
}  // namespace gbr

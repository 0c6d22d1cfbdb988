// gbr_kernels.h -- host-side launchers of the frame kernels (gbr_kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include "gbr_device.cuh"

namespace gbr {

// Programmatic dependent launch (sm_90+): a kernel started with launch_pdl
// may be scheduled while the kernel before it in the stream is finishing;
// it calls pdl_wait() before it touches anything, which returns once that
// kernel has completed and its writes are visible.  A kernel calls
// pdl_release() when its own work is issued, letting the next one launch.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Resident CTAs per SM of the raster kernels of a single frame with bins of
// bw x bh pixels.  ctas: the variant compiled for 2..6 CTAs per SM (0:
// default).
struct RasterGrid {
    int block64 = 1, block128 = 1, block512 = 1;   // block raster, by threads a CTA
    int record = 1;                   // record raster (bulk-copy staging)
    int& block(uint32_t threads) { return threads == 64u ? block64 : threads == 128u ? block128 : block512; }
    int block(uint32_t threads) const { return threads == 64u ? block64 : threads == 128u ? block128 : block512; }
};
cudaError_t raster_configure(uint32_t bw, uint32_t bh, uint32_t ctas, RasterGrid* per_sm);
// The block raster (gbr_raster.cu) for a batch frame (B's scenes) or a single
// frame (F), in CTAs of 64, 128 or 256 threads (a batch) or of 64, 128 or 512
// (a frame).
cudaError_t block_raster_configure(uint32_t bw, uint32_t bh, bool batch, uint32_t threads, uint32_t ctas,
                                   int* blocks_per_sm);
// Entries that a pass of such CTAs sorts where a pass size of `stage` is asked
// for (0: the most).
uint32_t block_raster_pass(uint32_t stage, uint32_t threads);
cudaError_t launch_block_raster(const FrameDev& F, const BatchDev& B, bool batch, uint32_t threads, uint32_t ctas,
                                uint32_t bw, uint32_t bh, uint32_t grid, cudaStream_t s);
// one: the mesh of a frame of one mesh (null otherwise)
cudaError_t launch_setup(const FrameDev& F, const MeshDev* one, bool predicted, cudaStream_t s);
// The bin scan of a frame (mode: kScanExact, ...), one launch.
ScanDev scan_of(const FrameDev& F, uint32_t mode);
uint32_t scan_blocks(uint32_t num_bins);   // tiles of 1024 bins
cudaError_t launch_scan(const ScanDev& S, cudaStream_t s);
cudaError_t launch_fill(const FrameDev& F, cudaStream_t s);
// Zeros the frame's list entries ahead of a scattering fill pass (see
// list_touch_kernel); worth its launch once a frame holds ~1M entries.
constexpr unsigned long long kListTouchMinPairs = 1ull << 20;
cudaError_t launch_list_touch(const FrameDev& F, cudaStream_t s);
cudaError_t launch_raster(const FrameDev& F, const RasterGrid& per_sm, cudaStream_t s);
// one: the mesh and lights of a frame of one mesh (null otherwise)
cudaError_t launch_shade(const FrameDev& F, const ShadeOne* one, cudaStream_t s);
cudaError_t launch_clear(const FrameDev& F, cudaStream_t s);

// Grid sizes of a batch frame (see BatchDev).
struct BatchLaunch {
    uint32_t tri_blocks;    // setup / fill blocks of all scenes
    uint32_t px_blocks;     // shade blocks of all scenes
    uint32_t raster_grid;   // persistent raster CTAs
    uint32_t raster_ctas;   // raster variant (CTAs per SM it is compiled for; 0: default)
    uint32_t raster_threads;   // raster CTA width: 128 or 256
    uint32_t bin_w, bin_h;  // the largest bin of the batch (shared-memory tile)
    ScanDev scan;           // the scan over the bins of every scene
};
// reset, setup + count, bin scan (three launches), fill, raster, shade
cudaError_t launch_batch(const BatchDev& B, const BatchLaunch& L, cudaStream_t s);

// Message returned by gbr_last_error_string() on the calling thread.
void set_last_error(const char* msg);

}  // namespace gbr

// gbr_kernels.cu -- the frame hot path on sm_103a.
//
//   setup_kernel : vertex stage (positions) + triangle assembly + cull +
//                  frustum reject + raster setup + depth-key bound + bin
//                  rectangle, and the count pass of exact binning (one
//                  atomic per (triangle, bin) pair, whose return -- the pair's
//                  rank in its bin -- is kept).
//   setup_rows_kernel: the same with block-private counter rows (dense
//                  frames): pairs counted per bin in shared memory, one
//                  global atomic per (block, bin) reserves the block's run.
//   scan_kernel  : (gbr_scan.cu) bin counts -> list offsets and raster work
//                  items (bin, chunk of its ids); frames of at most
//                  kFusedBins bins do it in the fill pass (fused_scan).
//   list_touch_kernel: zeros the frame's list entries in whole words so the
//                  fill's scattered stores merge in L2 (frames of >= 2^20
//                  pairs).
//   fill_kernel  : second pass: each pair's id goes to its bin's offset +
//                  rank, no atomics (fill_rows_kernel: to the block's run,
//                  slots from shared-memory cursors).
//   block_raster_kernel (gbr_raster.cu): persistent CTAs pull work items,
//                  depth-sort the chunk by the key bounds and rasterise it
//                  front to back, a warp to 8x4 pixels (frames of small
//                  triangles: the set-up pass has rasterised those itself);
//                  raster_kernel, here, takes the bulk-copy staging on request.
//   shade_kernel : each pixel's winner shaded once: colour, depth and id.
//
// Reference stages replaced: VS_Kernel, TA_Kernel, TB_Kernel,
// RA_PerTileKernel, PS_Kernel and the CLEAR_* kernels
// (CustomCUDARasterizer/CUDARenderer.cu:598-1129, launchers :1625-1966).
#include <algorithm>
#include <cstring>

#include "gbr_device.cuh"
#include "gbr_kernels.h"
#include "gbr_raster.cuh"
#include "gbr_shade.cuh"

namespace gbr {

static int sm_count() {
    static int sms = 0;
    if (sms <= 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            sms = 152;
        }
    }
    return sms;
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ uint32_t find_mesh(const FrameDev& F, uint32_t prim) {
    uint32_t lo = 0, hi = F.num_meshes - 1u;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (__ldg(&F.meshes[mid].prim_base) <= prim) lo = mid; else hi = mid - 1u;
    }
    return lo;
}

// Lower bound of the depth keys any fragment of the triangle can produce.
// A pixel covered under the 16.16 rule is at most the snapping distance
// outside the float triangle, so each float edge value there is at least
// -beta with beta <= 3*2^-17*D + 2^-32 + 2^-20*D^2 (D = the triangle's
// x + y extent; snapping moves vertices <= 2^-17 px; the float evaluation
// errs by <= 4 ulp of its product terms), and the three edge values sum to
// the float area within 2^-20*D^2 each.  With g = (2^-15*D + 2^-32 +
// 2^-18*D^2)/area, every weight is >= -g and the weights sum to 1 +- g, so
// z >= zmin*(1-g) - (3g + 2^-22)*max|z_i| when zmin >= 0 (2^-22 covers the
// rounding of the fused z chain).  The key of that bound never exceeds the
// key of a fragment of the triangle, so the triangle cannot win a pixel whose
// stored key is below it.  0: no bound (float path, vertices behind z = 0);
// 0x7FFFFFFF: every fragment has z >= 1 and loses everywhere.
__device__ __forceinline__ uint32_t hiz_key(const TriSetup& t) {
    if (t.mesh & kFlagFloat) return 0u;
    const float zmin = fminf(t.z0, fminf(t.z1, t.z2));
    if (!(zmin >= 0.f)) return 0u;
    const float zabs = fmaxf(fabsf(t.z0), fmaxf(fabsf(t.z1), fabsf(t.z2)));
    const float D = (max3f(t.x0, t.x1, t.x2) - min3f(t.x0, t.x1, t.x2)) + (max3f(t.y0, t.y1, t.y2) - min3f(t.y0, t.y1, t.y2)) + 1.f;
    const float g = (D * 3.0517578125e-05f + 2.3283064365386963e-10f + D * D * 3.814697265625e-06f) * t.inv_area;
    const float zb = zmin * (1.f - g) - (3.f * g + 2.384185791015625e-07f) * zabs;
    if (!(zb > 0.f)) return 0u;
    if (zb >= 1.f) return 0x7FFFFFFFu;
    return (uint32_t)__float2int_rz(__fmul_rn(zb, 2147483648.0f));
}

// One lane's raster of a small triangle with bin rectangle r, straight into
// the merge buffer: the raster's pixel box, exact edge functions, weights,
// depth and (key, id) minimum.  Returns false, having done nothing, for a box
// of more than kDirectPixels pixels.
__device__ __forceinline__ bool raster_direct(const FrameDev& F, const TriSetup& t, uint32_t prim, int4 r, int X0, int Y0,
                                              int X1, int Y1, int X2, int Y2) {
    // covered pixels lie in [ceil(min), floor(max)] of the snapped triangle,
    // and only those of its bins are rasterised
    const int px0 = max((min(X0, min(X1, X2)) + 0xFFFF) >> kFxBits, r.x * (int)F.bw);
    const int px1 = min(max(X0, max(X1, X2)) >> kFxBits, min((r.z + 1) * (int)F.bw, (int)F.width) - 1);
    const int py0 = max((min(Y0, min(Y1, Y2)) + 0xFFFF) >> kFxBits, r.y * (int)F.bh);
    const int py1 = min(max(Y0, max(Y1, Y2)) >> kFxBits, min((r.w + 1) * (int)F.bh, (int)F.height) - 1);
    if (px0 > px1 || py0 > py1) return true;
    if ((px1 - px0 + 1) * (py1 - py0 + 1) > kDirectPixels) return false;
    for (int y = py0; y <= py1; ++y)
        for (int x = px0; x <= px1; ++x) {
            const int fx = x << kFxBits, fy = y << kFxBits;
            if ((edge_fx(fx, fy, X0, Y0, X1 - X0, Y1 - Y0) | edge_fx(fx, fy, X1, Y1, X2 - X1, Y2 - Y1) |
                 edge_fx(fx, fy, X2, Y2, X0 - X2, Y0 - Y2)) < 0)
                continue;
            float w[3];
            weights_fixed(t, x, y, w);
            const float z = interp_z(w[0], w[1], w[2], t.z0, t.z1, t.z2);
            if (!(z >= 0.f && z < 1.f)) continue;   // as the raster rejects it
            const uint32_t key = (uint32_t)__float2int_rz(__fmul_rn(z, 2147483648.0f));
            atomicMin(F.gvis + ((size_t)y * F.width + (size_t)x), ((unsigned long long)key << 32) | prim);
        }
    return true;
}

// Vertex stage (positions), triangle assembly, cull, frustum reject, raster
// setup record, depth-key bound and bin rectangle of triangle `prim`, then the count pass
// (MODE 0), the predicted-capacity fill (MODE 1) or the count into the
// block's shared-memory row `s_row` (MODE 2).  Called by whole warps.
// Returns the warp's visible and float-path triangle counts (bits 0-15 and
// 16-31), for the block's statistics.
// `one`: the frame's only mesh (null: looked up).  DIRECT: small triangles
// are rasterised here (a variant of its own, for the registers), and MODE 2
// counts the triangles that the raster need not read in a row of their own.
template <int MODE, bool DIRECT = false>
__device__ __forceinline__ uint32_t setup_tri(const FrameDev& F, uint32_t prim, uint32_t walk, const MeshDev* one,
                                              uint32_t end, uint32_t* s_row = nullptr, uint32_t* s_skipped = nullptr) {
    const bool in_range = prim < end;
    uint2 rect = empty_rect();
    bool visible = false, fpath = false, skip = true;   // skip: the raster need not read the triangle's entries
    uint32_t key = 0u;
    if (in_range) {
        const uint32_t mi = one ? 0u : find_mesh(F, prim);
        const MeshDev& m = one ? *one : F.meshes[mi];
        uint32_t vid[3];
        tri_vertex_ids(m, prim - m.prim_base, vid);
        float nx[3], ny[3], nz[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const F3 p = fetch_position(m, vid[k]);
            const float4 c = xform_point(m.wvp, p.x, p.y, p.z);
            nx[k] = __fdiv_rn(c.x, c.w);
            ny[k] = __fdiv_rn(c.y, c.w);
            nz[k] = __fdiv_rn(c.z, c.w);
        }
        // culling (TA_Kernel, CUDARenderer.cu:759-777): BackFace and
        // FrontFace run the same test in the reference
        bool culled = false;
        if (F.cull != 2u) {
            const F3 a = f3(__fsub_rn(nx[1], nx[0]), __fsub_rn(ny[1], ny[0]), __fsub_rn(nz[1], nz[0]));
            const F3 b = f3(__fsub_rn(nx[2], nx[0]), __fsub_rn(ny[2], ny[0]), __fsub_rn(nz[2], nz[0]));
            const F3 n = normalize3(cross3(a, b));
            culled = dot3(f3(F.cam_fwd[0], F.cam_fwd[1], F.cam_fwd[2]), n) <= 0.0f;
        }
        // IsTriangleVisible (CUDAROPs.cu:168-178)
        const bool ax = (nx[0] < -1.f && nx[1] < -1.f && nx[2] < -1.f) || (nx[0] > 1.f && nx[1] > 1.f && nx[2] > 1.f);
        const bool ay = (ny[0] < -1.f && ny[1] < -1.f && ny[2] < -1.f) || (ny[0] > 1.f && ny[1] > 1.f && ny[2] > 1.f);
        const bool az = (nz[0] < 0.f && nz[1] < 0.f && nz[2] < 0.f) || (nz[0] > 1.f && nz[1] > 1.f && nz[2] > 1.f);
        visible = !culled && !ax && !ay && !az;
        if (visible) {
            const float2 s0 = to_screen(nx[0], ny[0], F.width, F.height);
            const float2 s1 = to_screen(nx[1], ny[1], F.width, F.height);
            const float2 s2 = to_screen(nx[2], ny[2], F.width, F.height);
            const int4 r = bin_rect(s0, s1, s2, F);
            const bool inside = fabsf(s0.x) < kGuardPx && fabsf(s0.y) < kGuardPx && fabsf(s1.x) < kGuardPx &&
                                fabsf(s1.y) < kGuardPx && fabsf(s2.x) < kGuardPx && fabsf(s2.y) < kGuardPx;
            float inv_area = 0.f;
            uint32_t flags;
            int X0 = 0, Y0 = 0, X1 = 0, Y1 = 0, X2 = 0, Y2 = 0;
            if (inside) {
                X0 = snap_fx(s0.x); Y0 = snap_fx(s0.y); X1 = snap_fx(s1.x);
                Y1 = snap_fx(s1.y); X2 = snap_fx(s2.x); Y2 = snap_fx(s2.y);
                // S = cross(v0 - v1, v2 - v1) of the snapped triangle: > 0 for the
                // covered winding (the three edge functions sum to S)
                const long long S = (long long)(X0 - X1) * (long long)(Y2 - Y1) -
                                    (long long)(Y0 - Y1) * (long long)(X2 - X1);
                // the float area the reference divides its weights by (CUDAROPs.cu:336)
                const float area = fabsf(__fmaf_rn(__fsub_rn(s0.x, s1.x), __fsub_rn(s0.y, s2.y),
                                                   -__fmul_rn(__fsub_rn(s0.y, s1.y), __fsub_rn(s0.x, s2.x))));
                skip = !(S > 0 && area > 0.f);
                inv_area = skip ? 0.f : __fdiv_rn(1.0f, area);
                flags = skip ? 0u : kFlagRaster;
            } else {
                fpath = true;
                skip = false;
                flags = kFlagFloat;
            }
            // the raster depth-sorts a bin's triangles by this bound before it
            // reads their records
            TriSetup t;
            t.x0 = s0.x; t.y0 = s0.y; t.x1 = s1.x; t.y1 = s1.y; t.x2 = s2.x; t.y2 = s2.y;
            t.z0 = nz[0]; t.z1 = nz[1]; t.z2 = nz[2]; t.inv_area = inv_area; t.mesh = mi | flags;
            key = hiz_key(t);
            uint4* rec = reinterpret_cast<uint4*>(F.setup) + 3u * (size_t)prim;
            rec[0] = make_uint4(__float_as_uint(s0.x), __float_as_uint(s0.y), __float_as_uint(s1.x), __float_as_uint(s1.y));
            rec[1] = make_uint4(__float_as_uint(s2.x), __float_as_uint(s2.y), __float_as_uint(nz[0]), __float_as_uint(nz[1]));
            rec[2] = make_uint4(__float_as_uint(nz[2]), __float_as_uint(inv_area), key, mi | flags);
            if (DIRECT && !skip && inside) skip = raster_direct(F, t, prim, r, X0, Y0, X1, Y1, X2, Y2);
            rect = pack_rect(r, skip);
            F.keys[prim] = key;
        }
        F.rects[prim] = rect;
    }
    const uint32_t counts = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, visible)) |
                            ((uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, fpath)) << 16);
    if (MODE == 0) bin_walk<0, DIRECT>(F, rect, 0u, visible, walk);
    else if (MODE == 2) count_rect(DIRECT && skip ? s_skipped : s_row, visible ? rect : empty_rect(), F.nbx, F.nby);
    else bin_walk<2>(F, rect, list_entry(prim, key, skip, F.key_mask), visible, walk);
    return counts;
}

// Frame statistics of a block: its warps' counts, summed in shared memory,
// then one atomic per counter and block (not per warp: every warp of the
// grid adding to the same two words serialises at one L2 slice).
__device__ __forceinline__ void add_block_stats(Ctl* ctl, uint32_t warp_vis, uint32_t warp_fp) {
    __shared__ uint32_t s_vis, s_fp;
    if (threadIdx.x == 0) { s_vis = 0u; s_fp = 0u; }
    __syncthreads();
    if ((threadIdx.x & 31u) == 0u) {
        if (warp_vis) atomicAdd(&s_vis, warp_vis);
        if (warp_fp) atomicAdd(&s_fp, warp_fp);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_vis) atomicAdd(&ctl->visible, s_vis);
        if (s_fp) atomicAdd(&ctl->float_path, s_fp);
    }
}

template <int MODE, bool ONE, bool DIRECT = false>
__global__ void __launch_bounds__(256) setup_kernel(FrameDev F, const __grid_constant__ MeshDev one) {
    pdl_wait();
    // predicted binning: the exact pass only runs after an overflow, and the
    // predicted pass stops once an overflow is known; neither runs after a
    // scan of the frame gave up (Ctl::overflow).  An exact frame starts here,
    // with nothing to check
    if (MODE == 1) {   // one answer for the whole block: blocks that run raise pred_overflow
        if (__syncthreads_or(F.ctl->overflow || F.ctl->pred_overflow)) return;
    } else if (F.exact_guard) {
        if (F.ctl->overflow || !F.ctl->pred_overflow) return;
    }
    // a resident grid strides over the triangles, so that a guarded launch
    // that does not run costs one wave of early exits
    uint32_t vis = 0, fp = 0;
    for (uint32_t base = blockIdx.x * blockDim.x; base < F.num_tris; base += gridDim.x * blockDim.x) {
        const uint32_t c = setup_tri<MODE, DIRECT>(F, base + threadIdx.x, (base + threadIdx.x) >> 5, ONE ? &one : nullptr, F.num_tris);
        vis += c & 0xFFFFu;
        fp += c >> 16;
    }
    add_block_stats(F.ctl, vis, fp);
    pdl_release();
}

// The bin scan inside the fill pass (F.fused_scan): every block scans all the
// bins' counts in its shared memory instead of waiting for a scan kernel's
// launch, its tiles' look-back and the offsets' way through memory.  A warp
// takes a contiguous range of 32-bin rows; row r's
// offsets and work items are written by block r mod grid, the totals by block
// 0.  Returns false for a frame that exceeds the storage (flagged, not
// filled).  The counts stay as they are, for the other blocks: the raster
// zeroes them.
template <uint32_t THREADS, bool DIRECT>
__device__ __forceinline__ bool fused_scan(const FrameDev& F, uint32_t* s_off) {
    constexpr uint32_t kWarps = THREADS / 32u;
    __shared__ unsigned long long s_a[kWarps], s_b[kWarps];
    __shared__ uint32_t s_base[kWarps];
    const uint32_t nb = F.num_bins, lane = lane_id(), warp = threadIdx.x >> 5, chunk = F.chunk;
    const uint32_t rows = (nb + 31u) / 32u, per = (rows + kWarps - 1u) / kWarps;
    const uint32_t r0 = min(warp * per, rows), r1 = min(r0 + per, rows);
    unsigned long long a = 0, b = 0;   // entries, work items
    uint32_t base = 0;                 // the last block, where items are smaller than base_chunk: those of that size
    const bool split = blockIdx.x == gridDim.x - 1u && chunk != F.base_chunk;
#pragma unroll 4
    for (uint32_t r = r0; r < r1; ++r) {
        const uint32_t i = r * 32u + lane;
        // c: entries the raster reads; c1 (DIRECT): the others
        const uint32_t c = i < nb ? F.counts[i] : 0u, c1 = i < nb && DIRECT ? F.counts[nb + i] : 0u;
        if (i < nb) {
            s_off[i] = c;
            if (DIRECT) s_off[nb + i] = c1;
            if (F.dirty && r % gridDim.x == blockIdx.x) F.dirty[i] = next_dirty(F.dirty[i], c + c1 != 0u);
        }
        a += (unsigned long long)c + c1;
        b += (c + chunk - 1u) / chunk;
        if (split) base += (c + F.base_chunk - 1u) / F.base_chunk;
    }
    if (split) base = __reduce_add_sync(0xFFFFFFFFu, base);
#pragma unroll
    for (uint32_t d = 16; d > 0; d >>= 1) {
        a += __shfl_xor_sync(0xFFFFFFFFu, a, d);
        b += __shfl_xor_sync(0xFFFFFFFFu, b, d);
    }
    if (lane == 0u) {
        s_a[warp] = a;
        s_b[warp] = b;
        if (split) s_base[warp] = base;
    }
    __syncthreads();
    unsigned long long total = 0, items = 0, at64 = 0, item64 = 0;
#pragma unroll 8
    for (uint32_t w = 0; w < kWarps; ++w) {
        if (w == warp) {
            at64 = total;
            item64 = items;
        }
        total += s_a[w];
        items += s_b[w];
    }
    const bool fits = total <= F.list_cap && items <= F.items_cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        F.ctl->num_pairs = total;
        F.ctl->num_items = fits ? (uint32_t)items : 0u;
        F.ctl->items_alloc = items;
        if (chunk == F.base_chunk) F.ctl->base_items[0] = (uint32_t)items;
        F.ctl->item_next = 0u;
        F.ctl->overflow = fits ? 0u : 1u;
        F.ctl->pred_overflow = F.ctl->error = F.ctl->num_sampled = F.ctl->shade_count = 0u;
        F.ctl->pred_capacity = 0ull;
        if (fits) F.offsets[nb] = (uint32_t)total;
    }
    if (split && threadIdx.x == 0) {
        for (uint32_t w = 1; w < kWarps; ++w) base += s_base[w];
        F.ctl->base_items[0] = base;
    }
    if (!fits) return false;
    uint32_t at = (uint32_t)at64, item = (uint32_t)item64;   // the totals fit 32 bits
    for (uint32_t r = r0; r < r1; ++r) {
        const uint32_t i = r * 32u + lane;
        const uint32_t c = i < nb ? s_off[i] : 0u, c1 = i < nb && DIRECT ? s_off[nb + i] : 0u;
        const uint32_t it = (c + chunk - 1u) / chunk;
        uint32_t x = c + c1, y = it;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, x, d), u = __shfl_up_sync(0xFFFFFFFFu, y, d);
            if (lane >= d) {
                x += t;
                y += u;
            }
        }
        const uint32_t start = at + x - c - c1;
        if (i < nb) {
            s_off[i] = start;
            if (DIRECT) s_off[nb + i] = start + c;
            if (r % gridDim.x == blockIdx.x) {
                F.offsets[i] = start;
                for (uint32_t k = 0; k < it; ++k)
                    F.items[item + y - it + k] = make_uint4(i, start + k * chunk, min(chunk, c - k * chunk), it);
            }
        }
        at += __shfl_sync(0xFFFFFFFFu, x, 31);
        item += __shfl_sync(0xFFFFFFFFu, y, 31);
    }
    __syncthreads();
    return true;
}

// The list entry of triangle `prim` with rectangle `rect`, in a fill pass.
__device__ __forceinline__ uint32_t rect_entry(const FrameDev& F, uint32_t prim, uint2 rect, bool in_range) {
    return list_entry(prim, in_range && F.key_mask ? F.keys[prim] : 0u, (rect.y & 0x80000000u) != 0u, F.key_mask);
}

// Second pass of exact binning for triangle `prim`.  Called by whole warps.
// s_off: the bins' offsets of a fused scan (MODE 4).
template <int MODE, bool DIRECT>
__device__ __forceinline__ void fill_tri(const FrameDev& F, uint32_t prim, uint32_t walk, const uint32_t* s_off = nullptr) {
    const bool in_range = prim < F.num_tris;
    const uint2 rect = in_range ? F.rects[prim] : empty_rect();
    bin_walk<MODE, DIRECT>(F, rect, rect_entry(F, prim, rect, in_range), in_range, walk, s_off);
}

template <bool DIRECT>
__global__ void __launch_bounds__(256) fill_kernel(FrameDev F) {
    pdl_wait();
    if (F.ctl->overflow || (F.exact_guard && !F.ctl->pred_overflow)) return;
    for (uint32_t base = blockIdx.x * blockDim.x; base < F.num_tris; base += gridDim.x * blockDim.x)
        fill_tri<1, DIRECT>(F, base + threadIdx.x, (base + threadIdx.x) >> 5);
    pdl_release();
}

// The same with the scan in it (at most kFusedBins bins, one counter a bin,
// or two in direct frames).
template <bool DIRECT>
__global__ void __launch_bounds__(256) fill_fused_kernel(FrameDev F) {
    __shared__ uint32_t s_off[(DIRECT ? 2u : 1u) * kFusedBins];
    pdl_wait();
    if (!fused_scan<256, DIRECT>(F, s_off)) return;
    for (uint32_t base = blockIdx.x * blockDim.x; base < F.num_tris; base += gridDim.x * blockDim.x)
        fill_tri<4, DIRECT>(F, base + threadIdx.x, (base + threadIdx.x) >> 5, s_off);
    pdl_release();
}

// Exact binning with block-private counter rows (num_bins <= kMaxRowBins,
// one kRowThreads block per SM, F.row_blocks blocks).  The count pass counts
// the block's pairs per bin in shared memory, then takes the block's run of
// each bin it touched with one global atomic per bin (blocks start their
// sweep at different bins, so the blocks' atomics on one bin do not arrive
// together); the run's start, relative to the bin, goes to the block's row
// of F.row_base.

// One run per bin the block touched: an atomic on the bin's counter each,
// `done(bin, count, start)` with its return.  Blocks start their sweep at
// different bins, and a thread's atomics are issued back to back.
template <typename Done>
__device__ __forceinline__ void reserve_runs(const uint32_t* counts, uint32_t nb, uint32_t* to, Done done) {
    const uint32_t shift = (uint32_t)(((unsigned long long)blockIdx.x * nb) / gridDim.x);
    for (uint32_t i0 = 0; i0 < nb; i0 += 8u * kRowThreads) {
        uint32_t bb[8], cc[8], rr[8];
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u) {
            const uint32_t i = i0 + u * kRowThreads + threadIdx.x;
            uint32_t b = i + shift;
            if (b >= nb) b -= nb;
            bb[u] = b;
            cc[u] = i < nb ? counts[b] : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u)
            if (cc[u]) rr[u] = atomicAdd(&to[bb[u]], cc[u]);
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u)
            if (cc[u]) done(bb[u], cc[u], rr[u]);
    }
}

// The block's triangles [first, end): an equal share each, in whole warps (a
// share in turns of kRowThreads left some blocks a turn more than others: 1M
// soup 176.2 -> 173.7 us a frame).  The count and the fill pass take the same.
__device__ __forceinline__ uint32_t row_share(const FrameDev& F, uint32_t& end) {
    const uint32_t per = ((F.num_tris + gridDim.x - 1u) / gridDim.x + 31u) & ~31u;
    const uint32_t first = min(blockIdx.x * per, F.num_tris);
    end = min(first + per, F.num_tris);
    return first;
}

// DIRECT: two rows, the second for entries that the raster need not read.
template <bool ONE, bool DIRECT>
__global__ void __launch_bounds__(kRowThreads, 1) setup_rows_kernel(FrameDev F, const __grid_constant__ MeshDev one) {
    extern __shared__ uint32_t s_row[];
    const uint32_t nb = F.num_bins, all = (DIRECT ? 2u : 1u) * nb;
    for (uint32_t b = threadIdx.x; b < all; b += blockDim.x) s_row[b] = 0u;
    __syncthreads();
    pdl_wait();
    uint32_t vis = 0, fp = 0, end;
    for (uint32_t base = row_share(F, end); base < end; base += kRowThreads) {
        const uint32_t c = setup_tri<2, DIRECT>(F, base + threadIdx.x, 0u, ONE ? &one : nullptr, end, s_row, s_row + nb);
        vis += c & 0xFFFFu;
        fp += c >> 16;
    }
    // the list's first touch_words words (the last frame's entries), zeroed
    // for the fill as list_touch_kernel does, by a pass whose memory
    // pipeline is otherwise idle
    uint4* const zero_to = reinterpret_cast<uint4*>(F.list);
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < F.touch_words; w += gridDim.x * blockDim.x)
        zero_to[w] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    prefix_2d(s_row, F.nbx, F.nby);
    if (DIRECT) prefix_2d(s_row + nb, F.nbx, F.nby);
    uint32_t* const row = F.row_base + (size_t)blockIdx.x * all;
    reserve_runs(s_row, all, F.counts, [&](uint32_t b, uint32_t, uint32_t at) { row[b] = at; });
    add_block_stats(F.ctl, vis, fp);
    pdl_release();
}

// The fill pass of block-private rows: the same blocks walk the same
// triangles; each bin's cursor starts at the bin's offset plus the block's
// run start, and every pair takes the next slot with a shared-memory atomic.
// Cursors of bins the block never touched hold unused values.
template <bool DIRECT>
__global__ void __launch_bounds__(kRowThreads, 1) fill_rows_kernel(FrameDev F) {
    extern __shared__ uint32_t s_row[];
    pdl_wait();
    const uint32_t all = (DIRECT ? 2u : 1u) * F.num_bins;
    const uint32_t* const row = F.row_base + (size_t)blockIdx.x * all;
    if (F.fused_scan) {
        if (!fused_scan<kRowThreads, DIRECT>(F, s_row)) return;
        for (uint32_t b = threadIdx.x; b < all; b += blockDim.x) s_row[b] += __ldg(row + b);
    } else {
        if (F.ctl->overflow) return;
        const uint32_t* const from = DIRECT ? F.sub_base : F.offsets;   // with one row a bin's entries start at its offset
        for (uint32_t b = threadIdx.x; b < all; b += blockDim.x) s_row[b] = __ldg(from + b) + __ldg(row + b);
    }
    __syncthreads();
    uint32_t end;
    for (uint32_t base = row_share(F, end); base < end; base += kRowThreads) {
        const uint32_t prim = base + threadIdx.x;
        const bool in_range = prim < end;
        const uint2 rect = in_range ? F.rects[prim] : empty_rect();
        fill_walk<DIRECT>(F, rect, rect_entry(F, prim, rect, in_range), s_row);
    }
    pdl_release();
}

// Predicted-capacity binning on block-private counter rows, in one launch:
// the count pass of setup_rows_kernel (setup + each pair counted in the
// block's shared-memory row), then one run per bin the block touched,
// reserved with a global atomic on the bin's cursor (which the capacity
// scan set to the bin's offset) and checked against the bin's end (offset +
// predicted capacity), then the fill pass of fill_rows_kernel over the same
// triangles, slots handed out from shared-memory cursors.  Against exact
// binning it saves the scan between count and fill and the second launch;
// against one returning global atomic per pair (setup_kernel<1>) it needs
// one per (block, bin).  A block whose run does not fit raises
// Ctl::pred_overflow and writes nothing (the exact kernels queued behind
// re-bin the frame); the other blocks' runs lie inside their capacities.
template <bool ONE, bool DIRECT>
__global__ void __launch_bounds__(kRowThreads, 1) predicted_rows_kernel(FrameDev F, const __grid_constant__ MeshDev one) {
    extern __shared__ uint32_t s_row[];
    __shared__ uint32_t s_ovf;
    pdl_wait();
    // one answer for the whole block: blocks that run raise pred_overflow, and
    // a block that started with some of its warps would count with rows that
    // nobody zeroed and store through them
    if (__syncthreads_or(F.ctl->overflow || F.ctl->pred_overflow)) return;
    const uint32_t nb = F.num_bins, tid = threadIdx.x;
    for (uint32_t b = tid; b < nb; b += kRowThreads) s_row[b] = 0u;
    if (tid == 0) s_ovf = 0u;
    __syncthreads();
    uint32_t vis = 0, fp = 0, end;
    const uint32_t first = row_share(F, end);
    for (uint32_t base = first; base < end; base += kRowThreads) {
        const uint32_t c = setup_tri<2, DIRECT>(F, base + tid, 0u, ONE ? &one : nullptr, end, s_row, s_row);
        vis += c & 0xFFFFu;
        fp += c >> 16;
    }
    __syncthreads();
    prefix_2d(s_row, F.nbx, F.nby);
    reserve_runs(s_row, nb, F.cursors, [&](uint32_t b, uint32_t c, uint32_t at) {
        if ((unsigned long long)at + c > __ldg(&F.bin_end[b])) {
            s_ovf = 1u;
            atomicOr(&F.ctl->pred_overflow, 1u);
        }
        s_row[b] = at;
    });
    __syncthreads();
    if (!s_ovf) {
        for (uint32_t base = first; base < end; base += kRowThreads) {
            const uint32_t prim = base + tid;
            const bool in_range = prim < end;
            const uint2 rect = in_range ? F.rects[prim] : empty_rect();
            fill_walk<false>(F, rect, rect_entry(F, prim, rect, in_range), s_row);
        }
    }
    add_block_stats(F.ctl, vis, fp);
    pdl_release();
}

// Zeros over the frame's bin-list entries [0, num_pairs) in whole 16-byte
// words, before the exact fill pass scatters its 4-byte stores there.  The
// list's sectors are then fully written in L2, and the scattered stores
// merge into them instead of each partly written sector being completed
// from DRAM (1M soup: scan + fill 84 -> 64 us with this pass).  The
// predicted fused pass, bound by its returning atomics, measured no gain.
__global__ void __launch_bounds__(256) list_touch_kernel(FrameDev F) {
    pdl_wait();
    if (!F.ctl->overflow) {
        const unsigned long long n = min((unsigned long long)F.ctl->num_pairs, F.list_cap);
        uint4* const p = reinterpret_cast<uint4*>(F.list);
        const unsigned long long words = (n + 3u) / 4u;   // list storage is 2 x list_cap entries
        for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < words;
             i += (unsigned long long)gridDim.x * blockDim.x)
            p[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    pdl_release();
}

cudaError_t launch_list_touch(const FrameDev& F, cudaStream_t s) {
    return launch_pdl(list_touch_kernel, dim3(4u * (uint32_t)sm_count()), dim3(256), 0, s, F);
}

// ---------------------------------------------------------------------------
// Raster + ROP + shade
// ---------------------------------------------------------------------------
struct RasterShared {
    TriSetup rec[kMaxPhase];     // setup records of the running phase
    uint32_t prim[kBatch];       // staged bin entries (rasterisable triangles)
    uint16_t order[kBatch];      // staged triangles, front to back by depth bucket
    uint32_t bucket[kDepthBuckets];   // counts -> starts -> (after the scatter) ends
    uint32_t warp_count[kRasterThreads / 32];
    uint32_t warp_max[kRasterThreads / 32];
    uint32_t item[4];
    __align__(16) uint4 item_next;   // the next work item, copied ahead by thread 0
    int next;
    __align__(8) unsigned long long rec_bar[2];   // mbarriers: a phase's setup records have landed (phases alternate)
};
static_assert(kDepthBuckets == kRasterThreads, "one depth bucket per thread");

// Setup records reach shared memory by bulk asynchronous copies (the TMA
// engine's cp.async.bulk, one 48-byte copy per record), each completing
// its bytes on one of the CTA's two mbarriers (phases alternate); readers
// wait for that barrier's parity.  Warp 0 issues a phase's copies while the
// phase before it rasterises, so they land in time.
constexpr uint32_t kRecWaitLimit = 1u << 22;   // polls before a wait gives up (the frame is flagged)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Warp 0 arms `bar` for `pn` records and copies the records of sorted
// entries [p0, p0 + pn) into their ring slots (entry k -> slot k mod
// kMaxPhase).
__device__ __forceinline__ void issue_records(TriSetup* rec, const TriSetup* setup, const uint32_t* prim,
                                              const uint16_t* order, uint32_t p0, uint32_t pn, uint32_t bar,
                                              uint32_t lane, uint32_t key_mask);

__device__ __forceinline__ void rec_copy(TriSetup* dst, const TriSetup* src, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 48, [%2];"
                 ::"r"(smem_addr(dst)), "l"(src), "r"(bar) : "memory");
}

__device__ __forceinline__ void issue_records(TriSetup* rec, const TriSetup* setup, const uint32_t* prim,
                                              const uint16_t* order, uint32_t p0, uint32_t pn, uint32_t bar,
                                              uint32_t lane, uint32_t key_mask) {
    if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(pn * 48u) : "memory");
    __syncwarp();
    for (uint32_t q = lane; q < pn; q += 32u) {
        const uint32_t k = p0 + q;
        rec_copy(&rec[k & (kMaxPhase - 1u)], setup + list_id(prim[order[k]], key_mask), bar);
    }
}

// Waits for phase `parity` of the mbarrier; false when the bound ran out.
__device__ __forceinline__ bool rec_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < kRecWaitLimit; ++it) {
        uint32_t done = 0;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// `key_bound` = hiz_key(t): a covered pixel whose stored key is already
// below it cannot be won by this triangle, and skips the weights and depth.
__device__ __forceinline__ void raster_fixed(const TriSetup& t, uint32_t prim, unsigned long long* tile, int tx0,
                                             int ty0, int tw, int th, uint32_t lane, uint32_t key_bound) {
    const int X0 = snap_fx(t.x0), Y0 = snap_fx(t.y0), X1 = snap_fx(t.x1);
    const int Y1 = snap_fx(t.y1), X2 = snap_fx(t.x2), Y2 = snap_fx(t.y2);
    const int minx = min(X0, min(X1, X2)), maxx = max(X0, max(X1, X2));
    const int miny = min(Y0, min(Y1, Y2)), maxy = max(Y0, max(Y1, Y2));
    // covered pixels lie in [ceil(min), floor(max)] of the snapped triangle
    const int px0 = max((minx + 0xFFFF) >> kFxBits, tx0), px1 = min(maxx >> kFxBits, tx0 + tw - 1);
    const int py0 = max((miny + 0xFFFF) >> kFxBits, ty0), py1 = min(maxy >> kFxBits, ty0 + th - 1);
    if (px0 > px1 || py0 > py1) return;
    const int bwid = px1 - px0 + 1;
    const int lsw = bwid <= 1 ? 0 : bwid <= 2 ? 1 : bwid <= 4 ? 2 : bwid <= 8 ? 3 : bwid <= 16 ? 4 : 5;
    const int sw = 1 << lsw, sh = 32 >> lsw;
    const int lx = (int)lane & (sw - 1), ly = (int)lane >> lsw;
    const int dxa = X1 - X0, dya = Y1 - Y0;
    const int dxb = X2 - X1, dyb = Y2 - Y1;
    const int dxc = X0 - X2, dyc = Y0 - Y2;
    // exact edge values at the lane's first pixel, then stepped by whole
    // stamps: E(x + sw, y) = E + sw * 2^16 * dy, E(x, y + sh) = E - sh * 2^16 * dx
    const int fx0 = (px0 + lx) << kFxBits, fy0 = (py0 + ly) << kFxBits;
    long long r2 = edge_fx(fx0, fy0, X0, Y0, dxa, dya);
    long long r0 = edge_fx(fx0, fy0, X1, Y1, dxb, dyb);
    long long r1 = edge_fx(fx0, fy0, X2, Y2, dxc, dyc);
    const long long stx = (long long)sw << kFxBits, sty = (long long)sh << kFxBits;
    const long long ix2 = stx * dya, ix0 = stx * dyb, ix1 = stx * dyc;
    const long long iy2 = -sty * dxa, iy0 = -sty * dxb, iy1 = -sty * dxc;
    for (int sy = py0; sy <= py1; sy += sh, r2 += iy2, r0 += iy0, r1 += iy1) {
        const int y = sy + ly;
        long long e2 = r2, e0 = r0, e1 = r1;
        for (int sx = px0; sx <= px1; sx += sw, e2 += ix2, e0 += ix0, e1 += ix1) {
            const int x = sx + lx;
            if (x > px1 || y > py1 || (e0 | e1 | e2) < 0) continue;
            unsigned long long* slot = tile + (y - ty0) * tw + (x - tx0);
            const unsigned long long cur = *((volatile unsigned long long*)slot);
            if ((uint32_t)(cur >> 32) < key_bound) continue;   // occluded: every fragment key is >= the bound
            float w[3];
            weights_fixed(t, x, y, w);
            const float z = interp_z(w[0], w[1], w[2], t.z0, t.z1, t.z2);
            // the reference rejects z < 0 or z > 1; z == 1 saturates the key to
            // INT_MAX and can never win the depth test (CUDAROPs.cu:343-345, 386)
            if (!(z >= 0.f && z < 1.f)) continue;
            const uint32_t key = (uint32_t)__float2int_rz(__fmul_rn(z, 2147483648.0f));
            const unsigned long long packed = ((unsigned long long)key << 32) | prim;
            if (packed < cur) atomicMin(slot, packed);   // a later, lower value only makes atomicMin a no-op
        }
    }
}

// Triangles outside the guard band: the reference's float edge functions.
__device__ __noinline__ void raster_float(const TriSetup& t, uint32_t prim, unsigned long long* tile, int tx0,
                                             int ty0, int tw, int th, uint32_t lane) {
    const float x0 = t.x0, y0 = t.y0, x1 = t.x1, y1 = t.y1, x2 = t.x2, y2 = t.y2;
    if (x0 != x0 || y0 != y0 || x1 != x1 || y1 != y1 || x2 != x2 || y2 != y2) return;
    int px0 = tx0, px1 = tx0 + tw - 1, py0 = ty0, py1 = ty0 + th - 1;
    const float fx0 = floorf(min3f(x0, x1, x2)) - 1.f, fx1 = ceilf(max3f(x0, x1, x2)) + 1.f;
    const float fy0 = floorf(min3f(y0, y1, y2)) - 1.f, fy1 = ceilf(max3f(y0, y1, y2)) + 1.f;
    if (fx0 > (float)px0) px0 = fx0 > (float)px1 ? px1 + 1 : (int)fx0;
    if (fx1 < (float)px1) px1 = fx1 < (float)px0 ? px0 - 1 : (int)fx1;
    if (fy0 > (float)py0) py0 = fy0 > (float)py1 ? py1 + 1 : (int)fy0;
    if (fy1 < (float)py1) py1 = fy1 < (float)py0 ? py0 - 1 : (int)fy1;
    if (px0 > px1 || py0 > py1) return;
    const int n = (px1 - px0 + 1) * (py1 - py0 + 1);
    const int wdt = px1 - px0 + 1;
    for (int i = (int)lane; i < n; i += 32) {
        const int x = px0 + i % wdt, y = py0 + i / wdt;
        float w[3];
        if (!weights_float(t, (float)x, (float)y, w)) continue;
        const float z = interp_z(w[0], w[1], w[2], t.z0, t.z1, t.z2);
        if (z < 0.f || z > 1.f) continue;  // NaN passes as in the reference
        const int k = cvt_s32(__fmul_rn(z, 2147483648.0f));
        if (k == 2147483647) continue;
        const unsigned long long packed = ((unsigned long long)(uint32_t)k << 32) | prim;
        unsigned long long* slot = tile + (y - ty0) * tw + (x - tx0);
        if (packed < *((volatile unsigned long long*)slot)) atomicMin(slot, packed);
    }
}

__device__ __forceinline__ void clear_pixel(const FrameDev& F, size_t gi) {
    F.colour[gi] = F.vis == 0u ? F.clear_colour32 : 0u;
    F.depth[gi] = 0.f;
    F.ids[gi] = kInvalidPrim;
}

// How a pass shades its winners: through the whole vertex stage and shader,
// from vertex colours (the winner's mesh looked up, or the frame's only one),
// or by depth.
enum ShadeKind { kShadeFull, kShadeFlat, kShadeFlatOne, kShadeDepth };

// Pixel (x, y), won by `prim`: the winner's weights and depth as the raster
// computed them, its colour, and the three outputs.  ONE: the frame's only
// mesh and its lights (null: looked up).
template <ShadeKind KIND>
__device__ __forceinline__ void resolve_pixel(const FrameDev& F, int x, int y, uint32_t prim, const ShadeOne* one = nullptr) {
    const size_t gi = (size_t)y * F.width + (size_t)x;
    const uint4* rp = reinterpret_cast<const uint4*>(F.setup) + 3u * (size_t)prim;
    const uint4 a = __ldg(rp), b = __ldg(rp + 1), c = __ldg(rp + 2);
    TriSetup t;
    t.x0 = __uint_as_float(a.x); t.y0 = __uint_as_float(a.y); t.x1 = __uint_as_float(a.z); t.y1 = __uint_as_float(a.w);
    t.x2 = __uint_as_float(b.x); t.y2 = __uint_as_float(b.y); t.z0 = __uint_as_float(b.z); t.z1 = __uint_as_float(b.w);
    t.z2 = __uint_as_float(c.x); t.inv_area = __uint_as_float(c.y); t.key = c.z; t.mesh = c.w;
    float w[3] = {0.f, 0.f, 0.f};
    if (t.mesh & kFlagFloat) weights_float(t, (float)x, (float)y, w);
    else weights_fixed(t, x, y, w);
    const float z = interp_z(w[0], w[1], w[2], t.z0, t.z1, t.z2);
    if (KIND == kShadeFlatOne) {   // needs no mesh lookup: the vertices load beside the record
        F.colour[gi] = shade_flat(F.one, prim, w);
    } else if (KIND == kShadeDepth) {
        F.colour[gi] = shade_depth(z);
    } else if (one) {
        F.colour[gi] = shade_fragment(F, one->mesh, one->lights, prim, w, z);
    } else {
        const MeshDev& m = F.meshes[t.mesh & kMeshMask];
        F.colour[gi] = KIND == kShadeFlat ? shade_flat(flat_mesh(m), prim - m.prim_base, w)
                                          : shade_fragment(F, m, F.lights, prim, w, z);
    }
    F.depth[gi] = z;
    F.ids[gi] = prim;
}

// The record raster, on request (GBR_STAGING_TMA): persistent CTAs that stage
// a phase's setup records in shared memory by bulk copies and merge
// fragments into a shared tile, a triangle to a warp.
template <int MIN_CTAS>
__global__ void __launch_bounds__(kRasterThreads, MIN_CTAS) raster_kernel(FrameDev F) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr uint32_t kEntries = kBatch, THREADS = kRasterThreads;
    RasterShared& S = *reinterpret_cast<RasterShared*>(smem_raw);
    unsigned long long* tile = reinterpret_cast<unsigned long long*>(smem_raw + sizeof(RasterShared));
    pdl_wait();
    Ctl* const Q = F.ctl;
    const uint4* const items = F.items;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    zero_counts(F);
    if (blockIdx.x == 0u && tid == 0u) close_counters(Q);
    if (Q->overflow) return;
    const uint32_t num_items = Q->num_items;
    const uint32_t phase = F.phase == 0u ? kPhase : min(F.phase, kMaxPhase);
    const uint32_t pass = F.stage == 0u ? kEntries : min(F.stage, kEntries);   // entries per raster pass
    // thread 0 runs one item ahead: the next item's queue slot is taken when
    // an item starts and its descriptor copied to shared memory
    // (asynchronously) while the item is staged
    uint32_t next_idx = 0;
    const uint32_t rec_bar0 = smem_addr(&S.rec_bar[0]);
    uint32_t rec_parity = 0;   // bit b: completions of record barrier b seen so far, mod 2
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(rec_bar0) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(rec_bar0 + 8u) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        next_idx = atomicAdd(&Q->item_next, 1u);
        fetch_item(&S.item_next, items, next_idx, num_items);
    }
    for (;;) {
        if (tid == 0) {
            cp_async_wait_all();
            const uint4 it = S.item_next;
            S.item[0] = it.x; S.item[1] = it.y; S.item[2] = it.z; S.item[3] = it.w;
            if (it.x != 0xFFFFFFFFu) next_idx = atomicAdd(&Q->item_next, 1u);
        }
        __syncthreads();
        const uint32_t bin = S.item[0];
        if (bin == 0xFFFFFFFFu) break;
        if (tid == 0) mark_drawn(F, bin);
        const uint32_t start = S.item[1], count = S.item[2], nchunks = S.item[3];
        const int tx0 = (int)((bin % F.nbx) * F.bw), ty0 = (int)((bin / F.nbx) * F.bh);
        const int tw = min((int)F.bw, (int)F.width - tx0), th = min((int)F.bh, (int)F.height - ty0);
        const int npx = (tw > 0 && th > 0) ? tw * th : 0;
        const uint32_t* const list = F.list;
        const TriSetup* const setup = F.setup;
        unsigned long long* const gvis = F.gvis;
        const uint32_t width = F.width;
        for (int i = (int)tid; i < npx; i += THREADS) tile[i] = kEmptyVis;
        if (tid == 0) fetch_item(&S.item_next, items, next_idx, num_items);
        const uint32_t* const keys = F.keys;
        const uint32_t key_mask = F.key_mask;
        for (uint32_t b0 = 0; b0 < count && npx > 0; b0 += pass) {
            // stage the entries with their depth-key bounds (no setup record
            // is read before a triangle's phase comes) and count the
            // rasterisable ones per depth bucket
            constexpr uint32_t kPer = kEntries / THREADS;
            const uint32_t n = min(pass, count - b0);
            __syncthreads();   // the previous batch is done with the shared arrays
            S.bucket[tid] = 0u;
            __syncthreads();
            // rows of THREADS entries up to the pass's n (uniform); entries at
            // or past n are never read
            const uint32_t rows = (n + THREADS - 1u) / THREADS;
#pragma unroll 4
            for (uint32_t j = 0; j < kPer; ++j) {
                if (j >= rows) break;
                const uint32_t idx = j * THREADS + tid;
                const uint32_t e = idx < n ? __ldg(list + start + b0 + idx) : kNoRasterBit;
                S.prim[idx] = e;
                if (!(e & kNoRasterBit)) atomicAdd(&S.bucket[entry_bucket(e, key_mask, keys)], 1u);
            }
            __syncthreads();
            // bucket starts: exclusive scan of the 256 counts; their sum is the
            // number of staged triangles
            uint32_t total = 0;
            {
                const uint32_t c = S.bucket[tid];
                uint32_t x = c;
#pragma unroll
                for (uint32_t d = 1; d < 32; d <<= 1) {
                    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, x, d);
                    if (lane >= d) x += t;
                }
                if (lane == 31u) S.warp_count[warp] = x;
                __syncthreads();
                uint32_t before = 0;
#pragma unroll
                for (uint32_t w = 0; w < THREADS / 32; ++w) {
                    const uint32_t wc = S.warp_count[w];
                    before += w < warp ? wc : 0u;
                    total += wc;
                }
                S.bucket[tid] = before + x - c;
            }
            __syncthreads();
#pragma unroll
            for (uint32_t j = 0; j < kPer; ++j) {
                if (j >= rows) break;
                const uint32_t idx = j * THREADS + tid;
                if (idx < n && !(S.prim[idx] & kNoRasterBit))
                    S.order[atomicAdd(&S.bucket[entry_bucket(S.prim[idx], key_mask, keys)], 1u)] = (uint16_t)idx;
            }
            // now S.bucket[b] = end of bucket b
            // phases of `phase` triangles; the tile's max depth key is refreshed
            // between phases.  A triangle whose key bound exceeds it cannot win
            // a pixel; once a whole bucket's lower bound does, the rest of the
            // batch is skipped.
            // phases of at most kMaxPhase / 2 triangles prefetch
            // the next phase's records into the other half of the ring
            const bool ahead = phase <= kMaxPhase / 2u;
            for (uint32_t p0 = 0, ph = 0; p0 < total; p0 += phase, ph ^= 1u) {
                __syncthreads();   // the order, or the previous phase's records and tile
                const uint32_t pn = min(phase, total - p0);
                const uint32_t bar = rec_bar0 + 8u * ph, bar_next = rec_bar0 + 8u * (ph ^ 1u);
                const bool next = ahead && p0 + phase < total;   // this phase prefetches the next one's records
                if (warp == 0) {
                    if (p0 == 0u || !ahead)   // this phase's records were not prefetched
                        issue_records(S.rec, setup, S.prim, S.order, p0, pn, bar, lane, key_mask);
                    if (next)
                        issue_records(S.rec, setup, S.prim, S.order, p0 + phase, min(phase, total - p0 - phase), bar_next,
                                      lane, key_mask);
                }
                if (b0 > 0 || p0 > 0) {
                    uint32_t m = 0;
                    for (int i = (int)tid; i < npx; i += THREADS)
                        m = max(m, (uint32_t)(tile[i] >> 32));
                    m = __reduce_max_sync(0xFFFFFFFFu, m);
                    if (lane == 0) S.warp_max[warp] = m;
                }
                if (tid == 0) S.next = (int)p0;
                __syncthreads();
                // every thread sees this phase's records land before any phase
                // decision; a phase that ends the batch early also waits for
                // the records it prefetched, so no copy is ever left in flight
                if (!rec_wait(bar, (rec_parity >> ph) & 1u) && tid == 0) atomicOr(&Q->error, 8u);
                rec_parity ^= 1u << ph;
                uint32_t tile_max = 0xFFFFFFFFu;
                if (b0 > 0 || p0 > 0) {
                    tile_max = 0;
#pragma unroll
                    for (uint32_t w = 0; w < THREADS / 32; ++w) tile_max = max(tile_max, S.warp_max[w]);
                }
                // buckets [0, tile_max >> kSortShift] can still hold a winner
                const uint32_t limit = tile_max >= 0x80000000u ? total : S.bucket[tile_max >> kSortShift];
                if (p0 >= limit) {   // uniform: every thread sees the same tile_max
                    if (next) {
                        if (!rec_wait(bar_next, (rec_parity >> (ph ^ 1u)) & 1u) && tid == 0) atomicOr(&Q->error, 8u);
                        rec_parity ^= 1u << (ph ^ 1u);
                    }
                    break;
                }
                const uint32_t p1 = min(limit, p0 + phase);
                for (;;) {   // a warp takes one sorted triangle at a time
                    int kb = 0;
                    if (lane == 0) kb = atomicAdd(&S.next, 1);
                    kb = __shfl_sync(0xFFFFFFFFu, kb, 0);
                    if (kb >= (int)p1) break;
                    const TriSetup& t = S.rec[(uint32_t)kb & (kMaxPhase - 1u)];
                    if (t.key > tile_max) continue;
                    const uint32_t prim = list_id(S.prim[S.order[kb]], key_mask);
                    if (t.mesh & kFlagFloat) raster_float(t, prim, tile, tx0, ty0, tw, th, lane);
                    else raster_fixed(t, prim, tile, tx0, ty0, tw, th, lane, t.key);
                }
            }
        }
        __syncthreads();
        // publish the tile: one chunk owns its pixels (plain stores); the
        // chunks of a longer bin merge with 64-bit atomicMin
        if (npx > 0 && count > 0) {
            for (int i = (int)tid; i < npx; i += THREADS) {
                const unsigned long long v = tile[i];
                unsigned long long* g = &gvis[(size_t)(ty0 + i / tw) * width + (size_t)(tx0 + i % tw)];
                if (nchunks == 1u) *g = v;
                else if (v != kEmptyVis) atomicMin(g, v);
            }
        }
        __syncthreads();
    }
}

// The thread's two pixels of tile (tx, ty): columns by 8 lanes, the second
// pixel half a tile below the first.
struct TilePixels {
    uint32_t x, y;
    unsigned long long v[2];   // their merge words
};
__device__ __forceinline__ TilePixels load_tile(const FrameDev& F, uint32_t tx, uint32_t ty, uint32_t y1) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    TilePixels p;
    p.x = tx * kTileW + (warp & 3u) * 8u + (lane & 7u);
    p.y = ty + (warp >> 2) * 4u + (lane >> 3);
#pragma unroll
    for (uint32_t k = 0; k < 2u; ++k) {
        const uint32_t yk = p.y + k * (kTileH / 2u);
        p.v[k] = p.x < F.width && yk < y1 ? F.gvis[(size_t)yk * F.width + p.x] : kEmptyVis;
    }
    return p;
}

// Shades a tile's pixels above row y1: the winners the raster left in the
// merge buffer (or the clear colour), and leaves the buffer empty for the
// next frame.  Both merge words are loaded before either pixel is shaded: the
// pass waits on the chain merge word -> record and vertices (2M soup at 4K:
// one pixel a thread 96 us, two 92, two with eight blocks an SM 82).
template <ShadeKind KIND>
__device__ __forceinline__ void shade_tile(const FrameDev& F, const TilePixels& p, uint32_t y1) {
    if (p.x >= F.width) return;
#pragma unroll
    for (uint32_t k = 0; k < 2u; ++k) {
        const uint32_t yk = p.y + k * (kTileH / 2u);
        if (yk >= y1) break;
        const size_t i = (size_t)yk * F.width + p.x;
        if (p.v[k] == kEmptyVis) {
            clear_pixel(F, i);
            continue;
        }
        F.gvis[i] = kEmptyVis;
        resolve_pixel<KIND>(F, (int)p.x, (int)yk, (uint32_t)p.v[k]);
    }
}

// One-pass shading: a block per tile, pixel rows [y0, y1).  With the mesh in
// the descriptor, colours converted without a table, reciprocals for
// divisions and 8x4 pixels to a warp, 2M soup at 4K 108 -> 82 us.
template <ShadeKind KIND>
__global__ void __launch_bounds__(256, KIND == kShadeFull ? 3 : KIND == kShadeFlat ? 6 : 8) shade_kernel(FrameDev F, uint32_t y0,
                                                                                                      uint32_t y1) {
    pdl_wait();
    const TilePixels p = load_tile(F, blockIdx.x, y0 + blockIdx.y * kTileH, y1);
    if (F.ctl->overflow) {   // a frame that was not rasterised, but for the set-up pass's small triangles
        for (uint32_t k = 0; k < 2u && F.direct; ++k)
            if (p.v[k] != kEmptyVis) F.gvis[(size_t)(p.y + k * (kTileH / 2u)) * F.width + p.x] = kEmptyVis;
        return;
    }
    shade_tile<KIND>(F, p, y1);
}

// Two-pass shading, for frames that shade through the full vertex stage
// (textured or lit meshes, the normal view).  The light pass clears the
// pixels no triangle won and queues the covered ones; the heavy pass shades
// the queue, 32 covered pixels to a warp, over the whole GPU.  In one pass
// a covered region's pixels sit a few to a warp inside blocks that keep
// their SM slot for the whole shading chain (4K icosphere: 140K covered
// pixels of 8.3M).
//
// Light pass: one thread per 4 consecutive pixels: their merge words come in with two
// 16-byte loads, an all-empty quad (most of a frame whose geometry covers a
// small part of the screen) is cleared with 16-byte stores, and a warp
// queues its covered pixels with one atomic.  Buffers not 16-byte aligned
// take per-pixel accesses.
__global__ void __launch_bounds__(256) shade_queue_kernel(FrameDev F) {
    // pixels [px_begin, px_end) (px_begin a multiple of 4)
    const uint32_t n = F.px_end ? F.px_end : F.width * F.height;
    pdl_wait();
    if (F.ctl->overflow) {
        // not rasterised: the buffers keep the last frame's pixels, and the
        // next frame must find those bins as they were
        if (F.dirty)
            for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < F.num_bins; b += gridDim.x * blockDim.x)
                if (F.dirty[b]) F.dirty[b] |= kDirtyNow;
        // what the set-up pass has drawn goes
        if (F.direct)
            for (uint32_t i = F.px_begin + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
                F.gvis[i] = kEmptyVis;
        return;
    }
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i0 = F.px_begin + (blockIdx.x * blockDim.x + threadIdx.x) * 4u;
    const bool aligned = ((reinterpret_cast<uintptr_t>(F.gvis) | reinterpret_cast<uintptr_t>(F.colour) |
                           reinterpret_cast<uintptr_t>(F.depth) | reinterpret_cast<uintptr_t>(F.ids)) & 15u) == 0u;
    // a quad whose pixels all lie in bins clean after the last frame and not
    // drawn in this one already holds the clear values (pixels outside the
    // bin grid are always written)
    bool live = i0 < n;
    if (F.dirty) {
        // the quad's row and column: one division per warp (its 32 quads
        // are consecutive), then at most one row wrap per lane on frames at
        // least 128 pixels wide
        uint32_t y = 0, x = 0;
        if (lane == 0u) {
            y = i0 / F.width;
            x = i0 - y * F.width;
        }
        y = __shfl_sync(0xFFFFFFFFu, y, 0);
        x = __shfl_sync(0xFFFFFFFFu, x, 0) + 4u * lane;
        if (F.width < 128u) {
            y = i0 / F.width;
            x = i0 - y * F.width;
        } else if (x >= F.width) {
            x -= F.width;
            ++y;
        }
        if (!live) {
        } else if (x + 3u < F.width && i0 + 3u < n) {   // one row: bins [x / bw, (x + 3) / bw] of bin row y / bh
            const bool p2 = ((F.bw & (F.bw - 1u)) | (F.bh & (F.bh - 1u))) == 0u;
            const uint32_t sx = (uint32_t)__ffs((int)F.bw) - 1u, sy = (uint32_t)__ffs((int)F.bh) - 1u;
            const uint32_t by = p2 ? y >> sy : y / F.bh;
            const uint32_t bx0 = p2 ? x >> sx : x / F.bw, bx1 = p2 ? (x + 3u) >> sx : (x + 3u) / F.bw;
            live = by >= F.nby || bx1 >= F.nbx;
            for (uint32_t bx = bx0; !live && bx <= bx1; ++bx)
                live = F.dirty[by * F.nbx + bx] != 0u;
        } else {   // a quad that wraps a row, or the frame's last pixels
            live = false;
            const uint32_t last = min(i0 + 3u, n - 1u);
            for (uint32_t i = i0; i <= last; ++i) {
                const uint32_t yi = i / F.width, xi = i - yi * F.width;
                const uint32_t bx = xi / F.bw, by = yi / F.bh;
                live |= bx >= F.nbx || by >= F.nby || F.dirty[by * F.nbx + bx] != 0u;
            }
        }
        if (!__any_sync(0xFFFFFFFFu, live)) return;   // the warp's 128 pixels already hold the clear values
    }
    uint32_t covered = 0;   // bit k: pixel i0 + k has a winner
    uint32_t won[4] = {0u, 0u, 0u, 0u};
    if (!live) {
    } else if (aligned && i0 + 4u <= n) {
        ulonglong2* g = reinterpret_cast<ulonglong2*>(F.gvis + i0);
        const ulonglong2 a = g[0], b = g[1];
        won[0] = (uint32_t)a.x; won[1] = (uint32_t)a.y; won[2] = (uint32_t)b.x; won[3] = (uint32_t)b.y;
        covered = (a.x != kEmptyVis ? 1u : 0u) | (a.y != kEmptyVis ? 2u : 0u) | (b.x != kEmptyVis ? 4u : 0u) |
                  (b.y != kEmptyVis ? 8u : 0u);
        if (covered == 0u) {
            const uint32_t c = F.vis == 0u ? F.clear_colour32 : 0u;
            *reinterpret_cast<uint4*>(F.colour + i0) = make_uint4(c, c, c, c);
            *reinterpret_cast<float4*>(F.depth + i0) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<uint4*>(F.ids + i0) = make_uint4(kInvalidPrim, kInvalidPrim, kInvalidPrim, kInvalidPrim);
        } else {   // the merge words are left empty for the next frame
            g[0] = g[1] = make_ulonglong2(kEmptyVis, kEmptyVis);
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k)
                if (!((covered >> k) & 1u)) clear_pixel(F, i0 + k);
        }
    } else {
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            if (i0 + k >= n) break;
            const unsigned long long v = F.gvis[i0 + k];
            if (v == kEmptyVis) {
                clear_pixel(F, i0 + k);
                continue;
            }
            covered |= 1u << k;
            won[k] = (uint32_t)v;
            F.gvis[i0 + k] = kEmptyVis;
        }
    }
    // the warp's covered pixels go to the queue in one run
    const uint32_t c = (uint32_t)__popc(covered);
    uint32_t incl = c;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += t;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (total) {
        uint32_t base = 0;
        if (lane == 31u) base = atomicAdd(&F.ctl->shade_count, total);
        base = __shfl_sync(0xFFFFFFFFu, base, 31);
        uint32_t at = base + incl - c;
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k)
            if ((covered >> k) & 1u) F.shade_list[at++] = make_uint2(i0 + k, won[k]);
    }
    pdl_release();
}

// 2 blocks per SM (<= 128 registers): the heavy pass is bound by the latency
// of a pixel's chain of dependent loads, and the registers keep the four
// maps' texels in flight (640x480 sphere frame 36.8 us with 4 blocks, 36.5
// with 3, 35.0 with 2; lit 4K icosphere-6 74.8, 75.8, 72.8; before the maps
// were fetched together, with the mesh looked up: 39.1 and 74.4).
// A pixel's chain is queue -> record and indices -> vertices -> texels: the
// queue holds the winner, a frame's only mesh comes by value (ONE), and the
// four maps are fetched together.
template <bool ONE>
__global__ void __launch_bounds__(256, 2) shade_list_kernel(FrameDev F, const __grid_constant__ ShadeOne one) {
    pdl_wait();
    if (F.ctl->overflow) return;
    const uint32_t count = F.ctl->shade_count;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
        const uint2 e = __ldg(F.shade_list + j);
        const uint32_t y = e.x / F.width;
        resolve_pixel<kShadeFull>(F, (int)(e.x - y * F.width), (int)y, e.y, ONE ? &one : nullptr);
    }
}

// Pixels no bin covers (num_bins * bin_dim smaller than the screen).
__global__ void clear_kernel(FrameDev F) {
    const size_t n = (size_t)F.width * F.height;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        F.colour[i] = F.vis == 0u ? F.clear_colour32 : 0u;
        F.depth[i] = 0.f;
        F.ids[i] = kInvalidPrim;
    }
}

// ---------------------------------------------------------------------------
// Batched frames: every stage of all scenes of a batch in one launch
// ---------------------------------------------------------------------------
static_assert(sizeof(Ctl) % 16 == 0, "control blocks are cleared as 16-byte words");

// Copies scene sc's frame descriptor into shared memory (whole block).
__device__ __forceinline__ void load_scene(const BatchDev& B, uint32_t sc, FrameDev& dst) {
    const uint4* src = reinterpret_cast<const uint4*>(B.scenes + sc);
    uint4* d = reinterpret_cast<uint4*>(&dst);
    for (uint32_t i = threadIdx.x; i < sizeof(FrameDev) / 16u; i += blockDim.x) d[i] = __ldg(src + i);
    __syncthreads();
}

__device__ __forceinline__ void clear_ctl(Ctl* c) {
    uint4* w = reinterpret_cast<uint4*>(c);
#pragma unroll
    for (uint32_t k = 0; k < sizeof(Ctl) / 16u; ++k) w[k] = make_uint4(0u, 0u, 0u, 0u);
}

// Clears the batch's control block and every scene's statistics block.
__global__ void batch_reset_kernel(BatchDev B) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) clear_ctl(B.ctl);
    if (i < B.num_scenes) clear_ctl(B.scenes[i].ctl);
}

// Block -> scene, then the scene's descriptor into shared memory.
// The batch's triangle and pixel passes are cut into chunks of 256 items,
// each belonging to one scene (B.tri_scene / B.px_scene).  A block walks a
// contiguous range of `per` chunks and reloads its shared-memory frame
// descriptor only when the scene changes (a scene's chunks are
// consecutive), so the descriptor copy and its barrier are paid per scene
// rather than per 256 items.  Walk ids stay those of the chunk (chunk * 8 +
// warp), so the count and fill passes meet the same rank slots whatever
// their ranges.
__device__ __forceinline__ bool enter_scene(const BatchDev& B, uint32_t sc, uint32_t& loaded, FrameDev& sF) {
    if (sc == loaded) return false;   // block-uniform
    __syncthreads();                  // every thread is done with the previous descriptor
    load_scene(B, sc, sF);
    loaded = sc;
    return true;
}

__global__ void __launch_bounds__(256) batch_setup_kernel(BatchDev B, uint32_t chunks, uint32_t per) {
    __shared__ __align__(16) FrameDev sF;
    const uint32_t c0 = blockIdx.x * per, c1 = min(c0 + per, chunks);
    uint32_t loaded = 0xFFFFFFFFu, vis = 0, fp = 0;
    pdl_wait();
    for (uint32_t v = c0; v < c1; ++v) {
        const uint32_t sc = __ldg(B.tri_scene + v);
        if (sc != loaded && loaded != 0xFFFFFFFFu) {   // the previous scene's statistics
            add_block_stats(sF.ctl, vis, fp);
            vis = fp = 0;
        }
        enter_scene(B, sc, loaded, sF);
        const uint32_t c = setup_tri<0>(sF, (v - __ldg(B.tri_blocks + sc)) * 256u + threadIdx.x,
                                        (v * 256u + threadIdx.x) >> 5, nullptr, sF.num_tris);
        vis += c & 0xFFFFu;
        fp += c >> 16;
    }
    if (loaded != 0xFFFFFFFFu) add_block_stats(sF.ctl, vis, fp);
    pdl_release();
}

// The fill pass keeps one block per chunk (a range loop measured slower
// here: 489 -> 653 us for the 256-soup batch, more registers per thread).
__global__ void __launch_bounds__(256) batch_fill_kernel(BatchDev B) {
    pdl_wait();
    if (B.ctl->overflow) return;
    __shared__ __align__(16) FrameDev sF;
    const uint32_t sc = __ldg(B.tri_scene + blockIdx.x);
    load_scene(B, sc, sF);
    fill_tri<1, false>(sF, (blockIdx.x - __ldg(B.tri_blocks + sc)) * 256u + threadIdx.x, (blockIdx.x * 256u + threadIdx.x) >> 5);
    pdl_release();
}

// KIND: every scene of the batch shades flat (B.all_flat), from one mesh, and
// the kernel holds only that path's registers; kShadeFull: each scene its own
// way.  The flat kinds were bound by L1 (91% busy: the descriptor's fields
// read from shared memory over and over, spilled registers); with its fields
// and the next tile's merge words in registers and four blocks an SM that do
// not spill, a batch frame of 32 uneven soups (26.3M pixels) takes 900 us
// (957 before; five blocks 904, six 912, without the words ahead 930).
template <ShadeKind KIND>
__global__ void __launch_bounds__(256, KIND == kShadeFull ? 3 : 4) batch_shade_kernel(BatchDev B, uint32_t chunks, uint32_t per) {
    pdl_wait();
    if (B.ctl->overflow) return;
    __shared__ __align__(16) FrameDev sF;
    const uint32_t c0 = blockIdx.x * per, c1 = min(c0 + per, chunks);
    uint32_t loaded = 0xFFFFFFFFu, tx = 0, ty = 0;
    TilePixels p;
    bool have = false;
    for (uint32_t v = c0; v < c1; ++v) {
        const uint32_t sc = __ldg(B.px_scene + v);
        if (enter_scene(B, sc, loaded, sF)) {
            const uint32_t tile = v - __ldg(B.px_blocks + sc), across = (sF.width + kTileW - 1u) / kTileW;
            ty = tile / across;
            tx = tile - ty * across;
            have = false;
        }
        // what the flat path reads of the descriptor, in registers: from
        // shared memory it is read again after every store
        const FrameDev F = sF;
        if (!have) p = load_tile(F, tx, ty * kTileH, F.height);
        const TilePixels cur = p;
        if (++tx * kTileW >= F.width) {   // a range's tiles follow one another
            tx = 0;
            ++ty;
        }
        // the next tile's merge words are on their way while this one is shaded
        have = KIND != kShadeFull && v + 1u < c1;
        if (have) p = load_tile(F, tx, ty * kTileH, F.height);
        if (KIND != kShadeFull) shade_tile<KIND>(F, cur, F.height);
        else if (sF.flat_shade) shade_tile<kShadeFlat>(sF, cur, sF.height);
        else shade_tile<kShadeFull>(sF, cur, sF.height);
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
// Blocks of 256 threads for a triangle pass: one per 256 triangles, at most
// 8 per SM.  The blocks stride over the triangles, so a guarded launch that
// does not run costs one grid of early exits; more blocks than are resident
// at once (the setup pass holds 5 per SM) balance uneven triangles better
// than exactly one wave (measured ~9% faster for the 1M soup).

static uint32_t triangle_blocks(uint32_t num_tris) {
    return std::min<uint32_t>((num_tris + 255u) / 256u, 8u * (uint32_t)sm_count());
}

// Dynamic shared memory of the block-row kernels: `rows` counters per bin (the
// opt-in above the default 48 KB is made once per device).
static cudaError_t row_smem(const FrameDev& F, uint32_t rows, size_t* bytes) {
    static uint64_t opted = 0;   // bit d: done on device d (devices 0..63)
    *bytes = (size_t)rows * F.num_bins * sizeof(uint32_t);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? (1ull << dev) : 0ull;
    if (!(opted & bit)) {
        const int most = (int)(kMaxRowBins * sizeof(uint32_t));
        e = cudaFuncSetAttribute(fill_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fill_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        for (auto* k : {setup_rows_kernel<true, false>, setup_rows_kernel<false, false>, setup_rows_kernel<true, true>,
                        setup_rows_kernel<false, true>, predicted_rows_kernel<true, true>, predicted_rows_kernel<true, false>,
                        predicted_rows_kernel<false, true>, predicted_rows_kernel<false, false>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return e;
        opted |= bit;
    }
    return cudaSuccess;
}

template <bool ONE>
static cudaError_t launch_setup(const FrameDev& F, const MeshDev& one, bool predicted, cudaStream_t s) {
    if (F.row_blocks) {
        size_t smem = 0;
        const cudaError_t e = row_smem(F, !predicted && F.direct ? 2u : 1u, &smem);
        if (e != cudaSuccess) return e;
        return launch_pdl(!predicted ? (F.direct ? setup_rows_kernel<ONE, true> : setup_rows_kernel<ONE, false>)
                          : F.direct ? predicted_rows_kernel<ONE, true>
                                     : predicted_rows_kernel<ONE, false>,
                          dim3(F.row_blocks), dim3(kRowThreads), smem, s, F, one);
    }
    const uint32_t blocks = triangle_blocks(F.num_tris);
    if (blocks == 0) return cudaSuccess;
    return launch_pdl(predicted ? (F.direct ? setup_kernel<1, ONE, true> : setup_kernel<1, ONE>)
                                : (F.direct ? setup_kernel<0, ONE, true> : setup_kernel<0, ONE>),
                      dim3(blocks), dim3(256), 0, s, F, one);
}

cudaError_t launch_setup(const FrameDev& F, const MeshDev* one, bool predicted, cudaStream_t s) {
    if (one) return launch_setup<true>(F, *one, predicted, s);
    MeshDev none;
    memset(&none, 0, sizeof none);
    return launch_setup<false>(F, none, predicted, s);
}

cudaError_t launch_fill(const FrameDev& F, cudaStream_t s) {
    if (F.row_blocks) {
        size_t smem = 0;
        const cudaError_t e = row_smem(F, F.direct ? 2u : 1u, &smem);
        if (e != cudaSuccess) return e;
        return launch_pdl(F.direct ? fill_rows_kernel<true> : fill_rows_kernel<false>, dim3(F.row_blocks), dim3(kRowThreads), smem, s, F);
    }
    const uint32_t blocks = triangle_blocks(F.num_tris);
    if (blocks == 0) return cudaSuccess;
    return launch_pdl(F.direct ? (F.fused_scan ? fill_fused_kernel<true> : fill_kernel<true>)
                               : (F.fused_scan ? fill_fused_kernel<false> : fill_kernel<false>),
                      dim3(blocks), dim3(256), 0, s, F);
}

static size_t record_smem(uint32_t bw, uint32_t bh) {
    return sizeof(RasterShared) + (size_t)bw * bh * sizeof(unsigned long long);
}

using RecordRaster = void (*)(FrameDev);

static RecordRaster record_variant(uint32_t ctas) {
    switch (ctas ? ctas : kDefaultRasterCtas) {
        case 2: return raster_kernel<2>;
        case 3: return raster_kernel<3>;
        case 5: return raster_kernel<5>;
        case 6: return raster_kernel<6>;
        default: return raster_kernel<4>;
    }
}

cudaError_t raster_configure(uint32_t bw, uint32_t bh, uint32_t ctas, RasterGrid* per_sm) {
    const size_t smem = record_smem(bw, bh);
    const RecordRaster k = record_variant(ctas);
    // the limit of the largest bins, whatever these are (as in block_raster_configure)
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)record_smem(kMaxBinDim, kMaxBinDim));
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm->record, k, kRasterThreads, smem);
    for (uint32_t threads : {64u, 128u, 512u})
        if (e == cudaSuccess) e = block_raster_configure(bw, bh, false, threads, ctas, &per_sm->block(threads));
    for (int* n : {&per_sm->record, &per_sm->block64, &per_sm->block128, &per_sm->block512}) *n = std::max(*n, 1);
    return e;
}

cudaError_t launch_raster(const FrameDev& F, const RasterGrid& per_sm, cudaStream_t s) {
    if (F.rec_tma)
        return launch_pdl(record_variant(F.raster_ctas), dim3((uint32_t)(sm_count() * per_sm.record)),
                          dim3(kRasterThreads), record_smem(F.bw, F.bh), s, F);
    BatchDev none;
    memset(&none, 0, sizeof none);
    return launch_block_raster(F, none, false, F.block_threads, F.raster_ctas, F.bw, F.bh,
                               (uint32_t)(sm_count() * per_sm.block(F.block_threads)), s);
}

cudaError_t launch_shade(const FrameDev& F, const ShadeOne* one, cudaStream_t s) {
    const dim3 b(256);
    if (!F.flat_shade && F.shade_list) {
        const uint32_t npx = (F.px_end ? F.px_end : F.width * F.height) - F.px_begin;
        const cudaError_t e = launch_pdl(shade_queue_kernel, dim3((npx + 1023u) / 1024u), b, 0, s, F);
        if (e != cudaSuccess) return e;
        // one resident wave: the queue is a few pixels per thread at most
        static int per_sm = 0;
        if (per_sm <= 0 &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, shade_list_kernel<true>, 256, 0) != cudaSuccess) {
            cudaGetLastError();
            per_sm = 2;
        }
        const dim3 g((uint32_t)std::max(per_sm, 1) * (uint32_t)sm_count());
        if (one) return launch_pdl(shade_list_kernel<true>, g, b, 0, s, F, *one);
        ShadeOne none;
        memset(&none, 0, sizeof none);
        return launch_pdl(shade_list_kernel<false>, g, b, 0, s, F, none);
    }
    const uint32_t y0 = F.row1 ? F.row0 * F.bh : 0u, y1 = F.row1 ? std::min(F.row1 * F.bh, F.height) : F.height;
    if (y0 >= y1) return cudaSuccess;   // a band below the screen
    const dim3 g((F.width + kTileW - 1u) / kTileW, (y1 - y0 + kTileH - 1u) / kTileH);
    if (F.flat_shade && F.one.vertices) return launch_pdl(shade_kernel<kShadeFlatOne>, g, b, 0, s, F, y0, y1);
    if (F.flat_shade) return launch_pdl(shade_kernel<kShadeFlat>, g, b, 0, s, F, y0, y1);
    if (F.vis == 1u) return launch_pdl(shade_kernel<kShadeDepth>, g, b, 0, s, F, y0, y1);
    return launch_pdl(shade_kernel<kShadeFull>, g, b, 0, s, F, y0, y1);
}

cudaError_t launch_batch(const BatchDev& B, const BatchLaunch& L, cudaStream_t s) {
    if (B.num_scenes == 0) return cudaSuccess;
    batch_reset_kernel<<<(B.num_scenes + 255u) / 256u, 256, 0, s>>>(B);
    // chunk ranges: about 16 blocks per SM, so the ranges balance over two
    // or more resident waves
    const uint32_t target = 16u * (uint32_t)sm_count();
    const uint32_t tri_per = std::max<uint32_t>(1u, (L.tri_blocks + target - 1u) / target);
    const uint32_t px_per = std::max<uint32_t>(1u, (L.px_blocks + target - 1u) / target);
    const uint32_t tri_grid = (L.tri_blocks + tri_per - 1u) / tri_per, px_grid = (L.px_blocks + px_per - 1u) / px_per;
    cudaError_t e = cudaSuccess;
    if (L.tri_blocks) e = launch_pdl(batch_setup_kernel, dim3(tri_grid), dim3(256), 0, s, B, L.tri_blocks, tri_per);
    if (e == cudaSuccess) e = launch_scan(L.scan, s);
    if (e == cudaSuccess && L.tri_blocks) e = launch_pdl(batch_fill_kernel, dim3(L.tri_blocks), dim3(256), 0, s, B);
    if (e != cudaSuccess) return e;
    FrameDev none;
    memset(&none, 0, sizeof none);
    e = launch_block_raster(none, B, true, L.raster_threads, L.raster_ctas, L.bin_w, L.bin_h, L.raster_grid, s);
    if (e != cudaSuccess) return e;
    if (L.px_blocks) {
        e = launch_pdl(B.all_flat == 2u ? batch_shade_kernel<kShadeFlatOne>
                       : B.all_flat     ? batch_shade_kernel<kShadeFlat>
                                        : batch_shade_kernel<kShadeFull>,
                       dim3(px_grid), dim3(256), 0, s, B, L.px_blocks, px_per);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

cudaError_t launch_clear(const FrameDev& F, cudaStream_t s) {
    clear_kernel<<<1024, 256, 0, s>>>(F);
    return cudaGetLastError();
}

}  // namespace gbr

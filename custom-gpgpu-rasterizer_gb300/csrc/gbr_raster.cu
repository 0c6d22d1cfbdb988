// gbr_raster.cu -- the block raster: the frame's default rasteriser.
//
// Persistent CTAs pull work items (a bin, or a chunk of a long bin's list).
// A CTA depth-sorts the item's entries by their key bounds and goes through
// them in phases of 32 triangles (128 in CTAs of 512 threads):
//   - a thread each, the phase's triangles are loaded, snapped and reduced to
//     three 32-bit edge values at the bin's first pixel (reduce_triangle);
//   - each warp owns blocks of 8x4 pixels of the bin, a pixel a lane (or
//     pairs of them, two pixels a lane: pixels_per_lane), whose
//     best (depth key, primitive) it keeps in registers.  It tests 32
//     triangles at once, a lane each, against the blocks (depth bound, box,
//     edges), then takes the ones that meet them one after another, every lane
//     testing its own pixels.
// A warp is done once the next triangle's depth bucket lies behind its
// blocks' farthest key, the item once every warp is.
//
// Why: a warp that sweeps a whole triangle over the bin pays the triangle's
// set-up (some 120 instructions) in all 32 lanes, steps 64-bit edge values
// and merges every fragment with a 64-bit shared-memory atomic; the kernel
// was bound by instruction issue.  Here a set-up is paid once per triangle
// and bin, the edge values are 32-bit, no pixel is shared between warps, and
// the depth cut works on 32 pixels instead of a bin's 256.
#include <algorithm>
#include <cstring>

#include "gbr_device.cuh"
#include "gbr_kernels.h"
#include "gbr_raster.cuh"

namespace gbr {

namespace {

constexpr int kBlockW = 8, kBlockH = 4;          // a warp's pixels
constexpr uint32_t kSortBuckets = 256u;          // depth buckets: the top 8 bits of the 31-bit key
constexpr int kEdgeClamp = 1 << 30;
// blk / nbw = blk * kInvBlocks[nbw] >> 10 for blk < 128, nbw <= 8 (a bin holds at most 8 x 16 blocks)
__device__ constexpr uint16_t kInvBlocks[9] = {0, 1025, 513, 342, 257, 205, 171, 147, 129};

// Entries depth-sorted at once, whatever smaller number is asked for: a pass
// costs its sort and barriers and reduces a phase of triangles that a longer
// one would have found to lie behind the block (batch of 32 uneven soups, CTAs
// of 128: passes of 32 entries 2916 us a frame, 128 1404, 512 953, 1024 897; 1M
// soup at 1080p: 64 587, 256 274, 512 212, 1024 179).
constexpr uint32_t kMinPass = 1024;

enum : uint32_t { kTriNarrow = 0u, kTriWide = 1u, kTriFloat = 2u };

// The phase's triangles reduced to the bin, every word an array over the
// phase:
//   a: edge values at the bin's first pixel (v0v1, v1v2, v2v0), primitive
//   b: dy, -dx of v0v1; dy, -dx of v1v2
//   c: dy, -dx of v2v0; key bound; pixel box in the bin (x0, x1, y0, y1, 6
//      bits each from bit 0, 8, 16, 24) and kind (bits 6, 7)
//   h: the upper halves of a wide triangle's 64-bit edge values (16, 16, 32
//      bits)
//   r: the setup record (screen x y, NDC z, 1 / area)
template <uint32_t P>
struct PhaseTris {
    uint4 a[P], b[P], c[P], r0[P], r1[P];
    uint2 r2[P], h[P];
};

// CTAs of 64, 128 or 256 threads fill the SM; those of 512 run frames of few
// items, whose time is that of their longest one: several warps share a
// block's triangles and a phase holds more of them.
template <int THREADS>
struct BlockShared {
    static constexpr uint32_t kWarps = THREADS / 32u;
    static constexpr uint32_t kEntries = THREADS <= 128 ? 8u * THREADS : 2048u;   // entries depth-sorted at once
    static constexpr uint32_t kPhase = THREADS == 512 ? 128u : 32u;        // triangles reduced at once
    PhaseTris<kPhase> tri;
    uint32_t sorted[kEntries];              // staged entries, front to back by bucket
    uint32_t hist[2][kSortBuckets];         // entries per bucket; passes alternate, each zeroed after its scan
    uint32_t start[kSortBuckets + 4u];      // first sorted entry of each bucket, then the total
    uint32_t item[2][6];                    // the running item (items alternate): bin, list start, count, chunks; x, y
    uint32_t scene[2];                      // batch: its scene
    uint32_t scene_loaded;                  // batch: scene whose descriptor `frame` holds
    __align__(16) uint4 item_next;          // the next work item, copied ahead by thread 0
    __align__(16) FrameDev frame;
};

// The edge value of an edge (a, d = b - a, 16.16) at the bin's first pixel
// (fx, fy), in units of 2^-16 px^2 rounded down.  Pixel steps change the
// exact 2^-32 value by whole multiples of 2^16 (x steps by dy, y steps by
// -dx), so the sign at every pixel of the bin is the sign of the rounded
// value plus those steps, with nothing lost.
__device__ __forceinline__ long long bin_edge(int fx, int fy, int ax, int ay, int dx, int dy) {
    return edge_fx(fx, fy, ax, ay, dx, dy) >> kFxBits;
}
// The value of a narrow triangle's edge, whose steps across the bin stay
// below 2^30: clamped there, the sign holds.
__device__ __forceinline__ int narrow_edge(long long e) {
    return e >= kEdgeClamp ? kEdgeClamp : e <= -kEdgeClamp ? -kEdgeClamp : (int)e;
}

// Triangle `prim` reduced to the bin of tw x th pixels at (tx0, ty0), into
// slot `k` of the phase.  One that covers none of the bin's pixels gets an
// empty box.
template <uint32_t P>
__device__ __forceinline__ void reduce_triangle(const TriSetup* setup, uint32_t prim, int tx0, int ty0,
                                                int tw, int th, PhaseTris<P>& out, uint32_t k) {
    const uint4* rp = reinterpret_cast<const uint4*>(setup) + 3u * (size_t)prim;
    const uint4 r0 = __ldg(rp), r1 = __ldg(rp + 1), r2 = __ldg(rp + 2);
    const float x0 = __uint_as_float(r0.x), y0 = __uint_as_float(r0.y), x1 = __uint_as_float(r0.z);
    const float y1 = __uint_as_float(r0.w), x2 = __uint_as_float(r1.x), y2 = __uint_as_float(r1.y);
    long long qa = 0, qb = 0, qc = 0;
    int dxa = 0, dya = 0, dxb = 0, dyb = 0, dxc = 0, dyc = 0;
    int px0 = 0, px1 = tw - 1, py0 = 0, py1 = th - 1;
    uint32_t kind = kTriFloat;
    if (r2.w & kFlagFloat) {
        if (x0 != x0 || y0 != y0 || x1 != x1 || y1 != y1 || x2 != x2 || y2 != y2) px1 = -1;
    } else {
        const int X0 = snap_fx(x0), Y0 = snap_fx(y0), X1 = snap_fx(x1);
        const int Y1 = snap_fx(y1), X2 = snap_fx(x2), Y2 = snap_fx(y2);
        const int minx = min(X0, min(X1, X2)), maxx = max(X0, max(X1, X2));
        const int miny = min(Y0, min(Y1, Y2)), maxy = max(Y0, max(Y1, Y2));
        // covered pixels lie in [ceil(min), floor(max)] of the snapped triangle
        px0 = max(((minx + 0xFFFF) >> kFxBits) - tx0, 0);
        px1 = min((maxx >> kFxBits) - tx0, px1);
        py0 = max(((miny + 0xFFFF) >> kFxBits) - ty0, 0);
        py1 = min((maxy >> kFxBits) - ty0, py1);
        dxa = X1 - X0; dya = Y1 - Y0;
        dxb = X2 - X1; dyb = Y2 - Y1;
        dxc = X0 - X2; dyc = Y0 - Y2;
        const int fx = tx0 << kFxBits, fy = ty0 << kFxBits;
        qa = bin_edge(fx, fy, X0, Y0, dxa, dya);
        qb = bin_edge(fx, fy, X1, Y1, dxb, dyb);
        qc = bin_edge(fx, fy, X2, Y2, dxc, dyc);
        // steps across the bin's blocks, which may reach past its last pixels:
        // at most their width + height times the extent
        kind = kTriWide;
        const int span = ((tw + kBlockW - 1) & -kBlockW) + ((th + 2 * kBlockH - 1) & (-2 * kBlockH));
        if ((long long)max(maxx - minx, maxy - miny) * span < kEdgeClamp) {
            kind = kTriNarrow;
            qa = narrow_edge(qa);
            qb = narrow_edge(qb);
            qc = narrow_edge(qc);
        }
    }
    uint32_t box = 63u | (63u << 16);   // empty: x0 = y0 = 63, x1 = y1 = 0
    if (px0 <= px1 && py0 <= py1)
        box = (uint32_t)px0 | ((uint32_t)px1 << 8) | ((uint32_t)py0 << 16) | ((uint32_t)py1 << 24);
    out.a[k] = make_uint4((uint32_t)qa, (uint32_t)qb, (uint32_t)qc, prim);
    out.b[k] = make_uint4((uint32_t)dya, (uint32_t)-dxa, (uint32_t)dyb, (uint32_t)-dxb);
    out.c[k] = make_uint4((uint32_t)dyc, (uint32_t)-dxc, r2.z, box | (kind << 6));
    out.r0[k] = r0;
    out.r1[k] = r1;
    out.r2[k] = make_uint2(r2.x, r2.y);
    out.h[k] = make_uint2((uint32_t)(qa >> 32) & 0xFFFFu | (uint32_t)(qb >> 32) << 16, (uint32_t)(qc >> 32));
}

// The three edge values of phase triangle i at (x, y) in the bin, or-ed:
// negative where one of them is.  Wide triangles in 64 bits.
template <bool WIDE, uint32_t P>
__device__ __forceinline__ int edges_at(uint4 q, uint4 d, uint4 c, const PhaseTris<P>& tri, uint32_t i, int xa,
                                        int ya, int xb, int yb, int xc, int yc) {
    if (!WIDE)
        return ((int)q.x + xa * (int)d.x + ya * (int)d.y) | ((int)q.y + xb * (int)d.z + yb * (int)d.w) |
               ((int)q.z + xc * (int)c.x + yc * (int)c.y);
    const uint2 h = tri.h[i];
    const long long ea = (long long)(((unsigned long long)(uint32_t)((int)(h.x << 16) >> 16) << 32) | q.x);
    const long long eb = (long long)(((unsigned long long)(uint32_t)((int)h.x >> 16) << 32) | q.y);
    const long long ec = (long long)(((unsigned long long)h.y << 32) | q.z);
    const long long e = (ea + (long long)xa * (int)d.x + (long long)ya * (int)d.y) |
                        (eb + (long long)xb * (int)d.z + (long long)yb * (int)d.w) |
                        (ec + (long long)xc * (int)c.x + (long long)yc * (int)c.y);
    return (int)(e >> 32);
}

// Which of the R blocks of pixels [bx, bx + 7] x [by + 4 r, by + 4 r + 3] of
// the bin does phase triangle `k` meet, with a fragment possibly at or before
// key far[r]?  Its box overlaps the block's, and no edge is negative on the
// whole block.
template <int R, uint32_t P>
__device__ __forceinline__ void meets_blocks(const PhaseTris<P>& tri, uint32_t k, int bx, int by, const uint32_t (&far)[R],
                                             uint32_t& kind, uint32_t& key, bool (&hit)[R]) {
    const uint4 c = tri.c[k];
    key = c.z;
    const int x0 = (int)(c.w & 63u), x1 = (int)((c.w >> 8) & 63u), y0 = (int)((c.w >> 16) & 63u), y1 = (int)(c.w >> 24);
    kind = (c.w >> 6) & 3u;
    const int ex = bx + kBlockW - 1;
    bool some = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        hit[r] = c.z <= far[r] && x0 <= ex && x1 >= bx && y0 <= by + kBlockH * (r + 1) - 1 && y1 >= by + kBlockH * r;
        some |= hit[r];
    }
    if (!some || kind == kTriFloat) return;
    const uint4 q = tri.a[k], d = tri.b[k];
    const int xa = (int)d.x > 0 ? ex : bx, ya = (int)d.y > 0 ? by + kBlockH - 1 : by;
    const int xb = (int)d.z > 0 ? ex : bx, yb = (int)d.w > 0 ? by + kBlockH - 1 : by;
    const int xc = (int)c.x > 0 ? ex : bx, yc = (int)c.y > 0 ? by + kBlockH - 1 : by;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int dy = kBlockH * r;
        hit[r] = hit[r] && (kind == kTriNarrow ? edges_at<false>(q, d, c, tri, k, xa, ya + dy, xb, yb + dy, xc, yc + dy)
                                               : edges_at<true>(q, d, c, tri, k, xa, ya + dy, xb, yb + dy, xc, yc + dy)) >= 0;
    }
}

template <uint32_t P>
__device__ __forceinline__ TriSetup load_record(const PhaseTris<P>& tri, uint32_t i) {
    const uint4 a = tri.r0[i], b = tri.r1[i];
    const uint2 c = tri.r2[i];
    TriSetup t;
    t.x0 = __uint_as_float(a.x); t.y0 = __uint_as_float(a.y); t.x1 = __uint_as_float(a.z); t.y1 = __uint_as_float(a.w);
    t.x2 = __uint_as_float(b.x); t.y2 = __uint_as_float(b.y); t.z0 = __uint_as_float(b.z); t.z1 = __uint_as_float(b.w);
    t.z2 = __uint_as_float(c.x); t.inv_area = __uint_as_float(c.y); t.key = 0u; t.mesh = 0u;
    return t;
}

// A triangle outside the guard band at pixel (x, y): the reference's float
// edge functions within its box widened by a pixel; its depth key in `key`.
__device__ __forceinline__ bool covers_float(const TriSetup& t, int x, int y, uint32_t& key) {
    const float fx0 = floorf(min3f(t.x0, t.x1, t.x2)) - 1.f, fx1 = ceilf(max3f(t.x0, t.x1, t.x2)) + 1.f;
    const float fy0 = floorf(min3f(t.y0, t.y1, t.y2)) - 1.f, fy1 = ceilf(max3f(t.y0, t.y1, t.y2)) + 1.f;
    const float px = (float)x, py = (float)y;
    if (fx0 > px || fx1 < px || fy0 > py || fy1 < py) return false;
    float w[3];
    if (!weights_float(t, px, py, w)) return false;
    const float z = interp_z(w[0], w[1], w[2], t.z0, t.z1, t.z2);
    if (z < 0.f || z > 1.f) return false;   // NaN passes as in the reference
    const int k = cvt_s32(__fmul_rn(z, 2147483648.0f));
    key = (uint32_t)k;
    return k != 2147483647;
}

__device__ __forceinline__ void take(unsigned long long& best, uint32_t key, uint32_t prim) {
    const unsigned long long packed = ((unsigned long long)key << 32) | prim;
    if (packed < best) best = packed;
}

// The triangles of the phase (all narrow or all wide) that meet the warp's
// blocks, meet[r] those of block r, against the lane's pixels (x, y + 4 r),
// (lx, ly + 4 r) in the bin; best[r] the nearest (depth key, primitive) so
// far, far[r] the block's farthest key.  `key`: the bound of the
// lane's own triangle -- as a block closes, the triangles behind its `far` are
// dropped, which most of a phase's are (1M soup: 73 of 91 a bin).
// U triangles a turn: a turn is one chain of dependent operations, and two
// triangles' run side by side where few warps are there to fill the gaps.
template <int U, bool WIDE, int R, uint32_t P>
__device__ __forceinline__ void raster_fixed_tris(const PhaseTris<P>& tri, uint32_t k0, const uint32_t (&meet)[R], uint32_t key,
                                                  int x, int y, int lx, int ly, unsigned long long (&best)[R],
                                                  uint32_t (&far)[R]) {
    uint32_t mask = meet[0];
#pragma unroll
    for (int r = 1; r < R; ++r) mask |= meet[r];
    while (mask) {   // warp-uniform
        bool cov[U][R], covers[U], some = false;
        uint32_t i[U], prim[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool any = u == 0 || mask != 0u;   // an odd one's second: the first again, covering nothing
            i[u] = any ? k0 + (uint32_t)__ffs((int)mask) - 1u : i[0];
            mask &= mask - 1u;
            const uint4 q = tri.a[i[u]], d = tri.b[i[u]], c = tri.c[i[u]];
            prim[u] = q.w;
            covers[u] = false;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int yr = ly + kBlockH * r;
                // a stored key below the triangle's bound: no fragment of it can win
                cov[u][r] = any && edges_at<WIDE>(q, d, c, tri, i[u], lx, yr, lx, yr, lx, yr) >= 0 &&
                            c.z <= (uint32_t)(best[r] >> 32);
                covers[u] |= cov[u][r];
            }
            some |= covers[u];
        }
        if (!__any_sync(0xFFFFFFFFu, some)) continue;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!covers[u]) continue;
            const TriSetup t = load_record(tri, i[u]);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (!cov[u][r]) continue;
                float w[3];
                weights_fixed(t, x, y + kBlockH * r, w);
                const float z = interp_z(w[0], w[1], w[2], t.z0, t.z1, t.z2);
                // the reference rejects z < 0 or z > 1; z == 1 saturates the key to
                // INT_MAX and can never win the depth test (CUDAROPs.cu:343-345, 386)
                if (z >= 0.f && z < 1.f) take(best[r], (uint32_t)__float2int_rz(__fmul_rn(z, 2147483648.0f)), prim[u]);
            }
        }
        uint32_t keep = 0u;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            far[r] = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best[r] >> 32));
            keep |= meet[r] & __ballot_sync(0xFFFFFFFFu, key <= far[r]);
        }
        mask &= keep;
    }
}

// The same for triangles on the float path.
template <uint32_t P>
__device__ __noinline__ unsigned long long raster_float_tris(const PhaseTris<P>& tri, uint32_t k0, uint32_t mask, int x,
                                                             int y, unsigned long long best) {
    for (; mask; mask &= mask - 1u) {
        const uint32_t i = k0 + (uint32_t)__ffs((int)mask) - 1u;
        uint32_t key = 0u;
        if (covers_float(load_record(tri, i), x, y, key)) take(best, key, tri.a[i].w);
    }
    return best;
}

// Single frame (BATCH false): work items of F.  Batch (BATCH true): work
// items of all scenes of B; an item's scene is found from its global bin,
// and its frame descriptor is copied to shared memory when it differs from
// the previous item's.  MIN_CTAS counts CTAs of 256 threads: twice as many
// of 128 threads are resident (of 512, two).
// R: a lane's pixels, its warp's blocks below one another.
template <int MIN_CTAS, bool BATCH, int THREADS, int R>
__global__ void __launch_bounds__(THREADS, THREADS == 512 ? 2 : MIN_CTAS * (256 / THREADS)) block_raster_kernel(FrameDev F, BatchDev B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Shared = BlockShared<THREADS>;
    constexpr uint32_t kWarps = Shared::kWarps, kEntries = Shared::kEntries, kPhase = Shared::kPhase;
    constexpr int U = THREADS == 512 ? 2 : 1;
    Shared& S = *reinterpret_cast<Shared*>(smem_raw);
    unsigned long long* const tile = reinterpret_cast<unsigned long long*>(smem_raw + sizeof(Shared));
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t i = tid; i < 2u * kSortBuckets; i += THREADS) (&S.hist[0][0])[i] = 0u;
    pdl_wait();
    Ctl* const Q = BATCH ? B.ctl : F.ctl;
    const uint4* const items = BATCH ? B.items : F.items;
    if (!BATCH) {
        zero_counts(F);
        if (blockIdx.x == 0u && tid == 0u) close_counters(Q);
    } else {
        for (uint32_t i = blockIdx.x * THREADS + tid; i < B.num_scenes; i += gridDim.x * THREADS) {
            close_counters(B.scenes[i].ctl);
            atomicAdd(&Q->num_visible, B.scenes[i].ctl->num_visible);
        }
    }
    if (Q->overflow) return;
    const uint32_t num_items = Q->num_items;
    const uint32_t stage_req = BATCH ? B.stage : F.stage;
    // entries per raster pass, at least kMinPass
    const uint32_t pass = stage_req == 0u ? kEntries : max(min(stage_req, kEntries), min(kMinPass, kEntries));
    // the first items are the CTAs' own, the rest are taken in turn.  Thread
    // 0 runs one item ahead: the next item's queue slot is taken when an
    // item starts and its descriptor copied to shared memory meanwhile
    if (tid == 0) {
        S.scene_loaded = 0xFFFFFFFFu;
        fetch_item(&S.item_next, items, blockIdx.x, num_items);
    }
    uint32_t hist_at = 0u;   // the histogram of the next sorted pass
    const int lx = (int)(lane & (kBlockW - 1u)), ly = (int)(lane / kBlockW);
    for (uint32_t turn = 0u;; turn ^= 1u) {
        if (tid == 0) {
            cp_async_wait_all();
            uint4 it = S.item_next;
            if (BATCH && it.x != 0xFFFFFFFFu) {
                const uint32_t sc = __ldg(B.bin_scene + it.x);
                S.scene[turn] = sc;
                it.x -= __ldg(B.bin_base + sc);
            }
            if (!BATCH) {
                const uint32_t row = it.x / F.nbx;
                S.item[turn][4] = (it.x - row * F.nbx) * F.bw;
                S.item[turn][5] = row * F.bh;
            }
            S.item[turn][0] = it.x; S.item[turn][1] = it.y; S.item[turn][2] = it.z; S.item[turn][3] = it.w;
            if (it.x != 0xFFFFFFFFu)
                fetch_item(&S.item_next, items, gridDim.x + atomicAdd(&Q->item_next, 1u), num_items);
        }
        __syncthreads();
        const uint32_t bin = S.item[turn][0];
        if (bin == 0xFFFFFFFFu) break;
        if (!BATCH && tid == 0) mark_drawn(F, bin);
        if (BATCH) {
            const uint32_t sc = S.scene[turn];
            if (sc != S.scene_loaded) {   // uniform across the CTA
                __syncthreads();          // every thread has compared
                const uint4* src = reinterpret_cast<const uint4*>(B.scenes + sc);
                uint4* dst = reinterpret_cast<uint4*>(&S.frame);
                for (uint32_t i = tid; i < sizeof(FrameDev) / 16u; i += THREADS) dst[i] = __ldg(src + i);
                if (tid == 0) S.scene_loaded = sc;
                __syncthreads();
            }
        }
        const FrameDev& G = BATCH ? S.frame : F;
        const uint32_t first = S.item[turn][1], count = S.item[turn][2], nchunks = S.item[turn][3];
        const uint32_t row = BATCH ? bin / G.nbx : 0u;
        const int tx0 = BATCH ? (int)((bin - row * G.nbx) * G.bw) : (int)S.item[turn][4];
        const int ty0 = BATCH ? (int)(row * G.bh) : (int)S.item[turn][5];
        const int tw = min((int)G.bw, (int)G.width - tx0), th = min((int)G.bh, (int)G.height - ty0);
        if (tw <= 0 || th <= 0) continue;   // a bin outside the screen (uniform)
        const uint32_t* const list = G.list;
        const TriSetup* const setup = G.setup;
        const uint32_t* const keys = G.keys;
        const uint32_t key_mask = G.key_mask;
        const uint32_t nbw = (uint32_t)(tw + kBlockW - 1) / kBlockW;
        const uint32_t nblk = nbw * ((uint32_t)(th + R * kBlockH - 1) / (R * kBlockH));   // R blocks as one
        const uint32_t inv = kInvBlocks[nbw];
        // a bin of fewer blocks than warps: `groups` warps share a block,
        // taking its triangles in turn and merging in the shared tile
        const uint32_t groups = nblk < kWarps ? kWarps / nblk : 1u, jobs = nblk * groups;
        for (uint32_t blk = warp; blk < nblk; blk += kWarps) {
            const uint32_t by = blk * inv >> 10, bx = blk - by * nbw;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                // pixels outside the bin: 0, which nothing beats
                const bool inside = (int)bx * kBlockW + lx < tw && (int)by * (R * kBlockH) + kBlockH * r + ly < th;
                tile[(blk * R + r) * 32u + lane] = inside ? kEmptyVis : 0ull;
            }
        }
        const bool direct = count <= min(kPhase, pass);   // one phase: nothing to sort
        for (uint32_t b0 = 0; b0 < count; b0 += pass) {
            const uint32_t n = min(pass, count - b0);
            uint32_t total = n;
            if (!direct) {
                // the entries that can cover a pixel, counted per depth
                // bucket: an entry's rank in its bucket is its place behind
                // the bucket's start
                constexpr uint32_t kPer = kEntries / THREADS;
                uint32_t* const hist = S.hist[hist_at];
                uint32_t e[kPer], place[kPer];
#pragma unroll
                for (uint32_t j = 0; j < kPer; ++j) {
                    e[j] = kNoRasterBit;
                    if (j * THREADS >= n) continue;   // uniform
                    const uint32_t idx = j * THREADS + tid;
                    if (idx < n) e[j] = __ldg(list + first + b0 + idx);
                }
#pragma unroll
                for (uint32_t j = 0; j < kPer; ++j) {
                    if (e[j] & kNoRasterBit) continue;
                    const uint32_t bucket = entry_bucket(e[j], key_mask, keys);
                    place[j] = (bucket << 16) | atomicAdd(&hist[bucket], 1u);
                }
                __syncthreads();   // also: every warp is done with the previous pass's order
                // bucket starts: every warp scans the whole histogram and
                // writes the same values, so no barrier follows
                {
                    const uint4 ca = *reinterpret_cast<const uint4*>(&hist[8u * lane]);
                    const uint4 cb = *reinterpret_cast<const uint4*>(&hist[8u * lane + 4u]);
                    const uint32_t mine = ca.x + ca.y + ca.z + ca.w + cb.x + cb.y + cb.z + cb.w;
                    uint32_t x = mine;
#pragma unroll
                    for (uint32_t d = 1; d < 32; d <<= 1) {
                        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, x, d);
                        if (lane >= d) x += t;
                    }
                    total = __shfl_sync(0xFFFFFFFFu, x, 31);
                    uint4 s;
                    s.x = x - mine; s.y = s.x + ca.x; s.z = s.y + ca.y; s.w = s.z + ca.z;
                    *reinterpret_cast<uint4*>(&S.start[8u * lane]) = s;
                    s.x = s.w + ca.w; s.y = s.x + cb.x; s.z = s.y + cb.y; s.w = s.z + cb.z;
                    *reinterpret_cast<uint4*>(&S.start[8u * lane + 4u]) = s;
                    if (lane == 0u) S.start[kSortBuckets] = total;
                }
                __syncwarp();
#pragma unroll
                for (uint32_t j = 0; j < kPer; ++j)
                    if (!(e[j] & kNoRasterBit)) S.sorted[S.start[place[j] >> 16] + (place[j] & 0xFFFFu)] = e[j];
                __syncthreads();
                for (uint32_t i = tid; i < kSortBuckets; i += THREADS) hist[i] = 0u;
                hist_at ^= 1u;
            }
            for (uint32_t p0 = 0; p0 < total; p0 += kPhase) {
                const uint32_t pn = min(kPhase, total - p0);
                if (tid < pn) {
                    const uint32_t entry = direct ? __ldg(list + first + b0 + tid) : S.sorted[p0 + tid];
                    if (entry & kNoRasterBit) S.tri.c[tid].w = 63u | (63u << 16);   // an empty box
                    else reduce_triangle(setup, list_id(entry, key_mask), tx0, ty0, tw, th, S.tri, tid);
                }
                __syncthreads();
                bool more = false;
                for (uint32_t w = warp; w < jobs; w += kWarps) {
                    const uint32_t group = groups > 1u ? w / nblk : 0u, blk = w - group * nblk;
                    const uint32_t brow = blk * inv >> 10;
                    const int bx = (int)(blk - brow * nbw) * kBlockW, by = (int)brow * (R * kBlockH);
                    const int px = bx + lx, py = by + ly;
                    unsigned long long* const slot = tile + blk * (R * 32u) + lane;
                    unsigned long long best[R];
                    uint32_t far[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        best[r] = *(volatile unsigned long long*)(slot + r * 32);
                        far[r] = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best[r] >> 32));
                    }
                    uint32_t limit = total;   // sorted entries from `limit` on lie in buckets behind every block's `far`
                    for (uint32_t c = 0; c < kPhase; c += 32u) {
                        const uint32_t farthest = R == 1 ? far[0] : max(far[0], far[R - 1]);
                        if (!direct && farthest < 0x80000000u) limit = S.start[(farthest >> kSortShift) + 1u];
                        if (c >= pn || p0 + c >= limit) break;
                        uint32_t kind = kTriNarrow, key = 0u, meet[R], narrow[R], any = 0u;
                        bool hit[R] = {};
                        if (c + lane < pn) meets_blocks<R>(S.tri, c + lane, bx, by, far, kind, key, hit);
                        // a group's share of the chunk, the same whatever its own `far`
                        const bool mine = groups == 1u || lane % groups == group;
#pragma unroll
                        for (int r = 0; r < R; ++r) any |= meet[r] = __ballot_sync(0xFFFFFFFFu, hit[r] && mine);
                        if (!any) continue;
                        const uint32_t other = __ballot_sync(0xFFFFFFFFu, kind != kTriNarrow);
#pragma unroll
                        for (int r = 0; r < R; ++r) narrow[r] = meet[r] & ~other;
                        raster_fixed_tris<U, false, R>(S.tri, c, narrow, key, tx0 + px, ty0 + py, px, py, best, far);
                        if (other & any) {
                            const uint32_t wide = __ballot_sync(0xFFFFFFFFu, kind == kTriWide);
#pragma unroll
                            for (int r = 0; r < R; ++r) narrow[r] = meet[r] & wide;
                            raster_fixed_tris<1, true, R>(S.tri, c, narrow, key, tx0 + px, ty0 + py, px, py, best, far);
#pragma unroll
                            for (int r = 0; r < R; ++r) {
                                const uint32_t rest = meet[r] & other & ~wide;
                                if (rest)
                                    best[r] = raster_float_tris(S.tri, c, rest, tx0 + px, ty0 + py + kBlockH * r, best[r]);
                                far[r] = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best[r] >> 32));
                            }
                        }
                    }
                    const uint32_t farthest = R == 1 ? far[0] : max(far[0], far[R - 1]);
                    if (!direct && farthest < 0x80000000u) limit = S.start[(farthest >> kSortShift) + 1u];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (groups > 1u) atomicMin(slot + r * 32, best[r]);
                        else slot[r * 32] = best[r];
                    }
                    more |= p0 + kPhase < limit;
                }
                // the phase's triangles are done with; on while some block is
                // not closed
                if (!__syncthreads_or(more)) break;
            }
        }
        if (count == 0u) __syncthreads();   // the tile's initial values
        // publish: one chunk owns its pixels (plain stores); the chunks of a
        // longer bin merge with 64-bit atomicMin, among themselves and with
        // what the set-up pass has drawn
        const bool own = nchunks == 1u && !G.direct;
        for (uint32_t blk = warp; blk < nblk; blk += kWarps) {
            const uint32_t by = blk * inv >> 10, bx = blk - by * nbw;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int x = (int)bx * kBlockW + lx, y = (int)by * (R * kBlockH) + kBlockH * r + ly;
                const unsigned long long best = tile[(blk * R + r) * 32u + lane];
                if (x >= tw || y >= th || best == kEmptyVis) continue;
                unsigned long long* g = &G.gvis[(size_t)(ty0 + y) * G.width + (size_t)(tx0 + x)];
                if (own) *g = best;
                else atomicMin(g, best);
            }
        }
    }
}

}  // namespace

size_t block_raster_smem(uint32_t bw, uint32_t bh, uint32_t threads) {
    const size_t shared = threads == 64u    ? sizeof(BlockShared<64>)
                          : threads == 128u ? sizeof(BlockShared<128>)
                          : threads == 256u ? sizeof(BlockShared<256>)
                                            : sizeof(BlockShared<512>);
    // an even number of rows, for pairs of blocks
    const size_t blocks = (size_t)((bw + kBlockW - 1) / kBlockW) * (((bh + kBlockH - 1) / kBlockH + 1u) & ~1u);
    return shared + blocks * 32u * sizeof(unsigned long long);
}

namespace {

using BlockRaster = void (*)(FrameDev, BatchDev);

template <bool BATCH, int THREADS, int R>
BlockRaster variant(uint32_t ctas) {
    switch (ctas ? ctas : kDefaultBlockCtas) {
        case 2: return block_raster_kernel<2, BATCH, THREADS, R>;
        case 3: return block_raster_kernel<3, BATCH, THREADS, R>;
        case 5: return block_raster_kernel<5, BATCH, THREADS, R>;
        case 6: return block_raster_kernel<6, BATCH, THREADS, R>;
        default: return block_raster_kernel<4, BATCH, THREADS, R>;
    }
}

// A lane's pixels: two where a bin has a pair of blocks for every warp (16x16
// bins and CTAs of 128 threads, say).  They read a triangle and step its edges
// once for both, and a pair of blocks goes through the tests and the tile's
// loads once (batch of 32 uneven soups, 32x32 bins: CTAs of 128 394M -> 335M
// instructions, frame 1005 -> 982 us, CTAs of 256 950 -> 907; 2M soup at 4K,
// 16x16 bins: 449 -> 443).  In smaller bins the pairs would leave warps to
// share one (the batch with CTAs of 256: 16x16 bins 1459 -> 1667, 8x8 4206 ->
// 4753), as in the frames of few items that CTAs of 512 run.
int pixels_per_lane(uint32_t bw, uint32_t bh, uint32_t threads) {
    const uint32_t pairs = ((bw + 7u) / 8u) * ((bh + 7u) / 8u);
    return threads != 512u && pairs >= threads / 32u ? 2 : 1;
}

BlockRaster variant(uint32_t bw, uint32_t bh, bool batch, uint32_t threads, uint32_t ctas) {
    const bool two = pixels_per_lane(bw, bh, threads) == 2;
    if (batch && threads == 64u) return variant<true, 64, 1>(ctas);   // bins of one or two blocks
    if (batch && threads != 128u) return two ? variant<true, 256, 2>(ctas) : variant<true, 256, 1>(ctas);
    if (batch) return two ? variant<true, 128, 2>(ctas) : variant<true, 128, 1>(ctas);
    if (threads == 512u) return block_raster_kernel<2, false, 512, 1>;
    if (threads == 64u) return two ? variant<false, 64, 2>(ctas) : variant<false, 64, 1>(ctas);
    return two ? variant<false, 128, 2>(ctas) : variant<false, 128, 1>(ctas);
}

}  // namespace

cudaError_t block_raster_configure(uint32_t bw, uint32_t bh, bool batch, uint32_t threads, uint32_t ctas,
                                   int* blocks_per_sm) {
    const BlockRaster k = variant(bw, bh, batch, threads, ctas);
    // the limit belongs to the kernel, not to the caller: always that of the
    // largest bins, so that no other renderer's launches are refused
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)block_raster_smem(kMaxBinDim, kMaxBinDim, threads));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k, (int)threads, block_raster_smem(bw, bh, threads));
}

// As the kernel reckons it (which calls no function for it: frames took 0.7%
// longer).
uint32_t block_raster_pass(uint32_t stage, uint32_t threads) {
    const uint32_t entries = threads == 64u    ? BlockShared<64>::kEntries
                             : threads == 128u ? BlockShared<128>::kEntries
                             : threads == 256u ? BlockShared<256>::kEntries
                                               : BlockShared<512>::kEntries;
    return stage == 0u ? entries : std::max(std::min(stage, entries), std::min(kMinPass, entries));
}

cudaError_t launch_block_raster(const FrameDev& F, const BatchDev& B, bool batch, uint32_t threads, uint32_t ctas,
                                uint32_t bw, uint32_t bh, uint32_t grid, cudaStream_t s) {
    return launch_pdl(variant(bw, bh, batch, threads, ctas), dim3(grid), dim3(threads), block_raster_smem(bw, bh, threads), s, F,
                      B);
}

}  // namespace gbr

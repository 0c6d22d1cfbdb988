// gbr_shade.cuh -- deferred per-pixel shading of the winning fragment.
//
// After visibility is resolved for a tile, each pixel's winning primitive is
// re-fetched, its three vertices go through the full vertex stage
// (GetNDCVertex, CustomCUDARasterizer/CUDAROPs.cu:99-118), the fragment
// attributes are interpolated as RasterizePixelAtomic does
// (CUDAROPs.cu:347-380) and the pixel shader of the selected
// VisualisationState runs (PS_Kernel / PS_VisualiseDepthColourKernel /
// PS_VisualiseNormalKernel, CUDARenderer.cu:833-897).  Only one fragment per
// pixel is shaded, instead of every fragment that wins a depth test.
#pragma once
#include "gbr_device.cuh"

namespace gbr {

// b / 255 for a byte value b, correctly rounded: the RGBA8 vertex colours and
// texels read as GetRGBColor (RGBRaw.h:34-38) divides.  The quotient estimate
// is corrected by its exact residual (Markstein); a product with 1/255 alone
// differs in 126 of the 256 values, this in none.  Four operations and no
// load: a table of the quotients cost a pixel nine scattered loads.
__device__ __forceinline__ float over255(uint32_t b) {
    const float x = (float)b, inv = 1.0f / 255.0f;
    const float q = __fmul_rn(x, inv);
    return __fmaf_rn(__fmaf_rn(-255.0f, q, x), inv, q);
}

struct OVtx {
    float px, py, pz, pw;  // NDC xyz, clip w
    float u, v;
    F3 n, tan, vd, c;
    F3 wp;                 // world position (scene lights)
};

__device__ __forceinline__ void fetch_full(const MeshDev& m, uint32_t vi, float iv[14]) {
    if (m.vertex_format == kVertexPos3Rgba8) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(m.vertices) + vi);
        const uint32_t rgba = __float_as_uint(v.w);
        iv[0] = v.x; iv[1] = v.y; iv[2] = v.z;
#pragma unroll
        for (int k = 3; k < 11; ++k) iv[k] = 0.f;
        // GetRGBColor (RGBRaw.h:34-38): r = byte0 / 255
        iv[11] = over255(rgba & 0xFFu);
        iv[12] = over255((rgba >> 8) & 0xFFu);
        iv[13] = over255((rgba >> 16) & 0xFFu);
    } else {
        const float2* b = reinterpret_cast<const float2*>(reinterpret_cast<const float*>(m.vertices) + 14u * (size_t)vi);
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const float2 t = __ldg(b + k);
            iv[2 * k] = t.x;
            iv[2 * k + 1] = t.y;
        }
    }
}

__device__ __forceinline__ OVtx vertex_stage(const MeshDev& m, const FrameDev& F, uint32_t vi) {
    float iv[14];
    fetch_full(m, vi, iv);
    OVtx o;
    const float4 clip = xform_point(m.wvp, iv[0], iv[1], iv[2]);
    o.px = __fdiv_rn(clip.x, clip.w);
    o.py = __fdiv_rn(clip.y, clip.w);
    o.pz = __fdiv_rn(clip.z, clip.w);
    o.pw = clip.w;
    o.n = rot3(m.world, f3(iv[5], iv[6], iv[7]));
    o.tan = rot3(m.world, f3(iv[8], iv[9], iv[10]));
    const float4 wp = xform_point(m.world, iv[0], iv[1], iv[2]);
    o.vd = normalize3(sub3(f3(wp.x, wp.y, wp.z), f3(F.cam_pos[0], F.cam_pos[1], F.cam_pos[2])));
    o.wp = f3(wp.x, wp.y, wp.z);
    o.u = iv[3];
    o.v = iv[4];
    o.c = f3(iv[11], iv[12], iv[13]);
    return o;
}

__device__ __forceinline__ F3 rgb_of(uint32_t c) {   // byte / 255 per channel
    return f3(over255(c & 0xFFu), over255((c >> 8) & 0xFFu), over255((c >> 16) & 0xFFu));
}

// A texture lookup in two halves, so that a pixel's four maps are all on
// their way before the first texel is converted: fetch() loads the texels
// (and keeps the bilinear fractions), colour() combines them.  SS: the
// sample state.
template <uint32_t SS>
struct Lookup {
    static constexpr int kTaps = SS == 0u ? 1 : SS == 1u ? 5 : 4;
    uint32_t c[kTaps];
    float ax, ay;
    bool in;

    __device__ __forceinline__ void fetch(const TexDev& t, float u, float v) {
        in = true;
        if (SS == 2u) {
            // bilinear filtering (the build's extension, GBR_SAMPLE_BILINEAR):
            // texel centres at (i + 1/2) / size, the four nearest texels
            // weighted by the fractional offsets, addresses clamped to the
            // texture
            const float x = __fmaf_rn(u, (float)t.w, -0.5f), y = __fmaf_rn(v, (float)t.h, -0.5f);
            const float fx = floorf(x), fy = floorf(y);
            ax = __fsub_rn(x, fx);
            ay = __fsub_rn(y, fy);
            const int w = (int)t.w, h = (int)t.h;
            int xi = cvt_s32(fx), yi = cvt_s32(fy);
            xi = xi < -1 ? -1 : (xi > w - 1 ? w - 1 : xi);
            yi = yi < -1 ? -1 : (yi > h - 1 ? h - 1 : yi);
            const uint32_t x0 = (uint32_t)(xi < 0 ? 0 : xi), x1 = (uint32_t)(xi + 1 > w - 1 ? w - 1 : xi + 1);
            const uint32_t y0 = (uint32_t)(yi < 0 ? 0 : yi), y1 = (uint32_t)(yi + 1 > h - 1 ? h - 1 : yi + 1);
            c[0] = __ldg(t.px + x0 + y0 * t.w);
            c[1 % kTaps] = __ldg(t.px + x1 + y0 * t.w);
            c[2 % kTaps] = __ldg(t.px + x0 + y1 * t.w);
            c[3 % kTaps] = __ldg(t.px + x1 + y1 * t.w);
            return;
        }
        // SamplePoint (CUDATextureSampler.cuh:87-104): u = int(uv.x*w + 0.5);
        // out of range samples magenta
        const int x = cvt_s32(__fmaf_rn(u, (float)t.w, 0.5f));
        const int y = cvt_s32(__fmaf_rn(v, (float)t.h, 0.5f));
        in = !(x < 0 || y < 0 || (uint32_t)x >= t.w || (uint32_t)y >= t.h);
        if (!in) return;
        if (SS == 0u) {
            c[0] = __ldg(t.px + (uint32_t)x + (uint32_t)y * t.w);
            return;
        }
        // SampleLinear (CUDATextureSampler.cuh:112-190): the centre and its
        // four row-major neighbours (wrapping across rows, clamped at the
        // buffer ends)
        const int size = (int)(t.w * t.h);
        const int o = x + y * (int)t.w;
        c[0] = __ldg(t.px + (o - 1 < 0 ? o : o - 1));
        c[1 % kTaps] = __ldg(t.px + (o + 1 >= size ? o : o + 1));
        c[2 % kTaps] = __ldg(t.px + (o + (int)t.w >= size ? o : o + (int)t.w));
        c[3 % kTaps] = __ldg(t.px + (o - (int)t.w < 0 ? o : o - (int)t.w));
        c[4 % kTaps] = __ldg(t.px + o);
    }

    __device__ __forceinline__ F3 colour() const {
        if (!in) return f3(1.f, 0.f, 1.f);
        float out[3];
        if (SS == 0u) {
            const F3 p = rgb_of(c[0]);
            out[0] = p.x; out[1] = p.y; out[2] = p.z;
        } else
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float a = (float)((c[0] >> (8 * k)) & 0xFFu), b = (float)((c[1 % kTaps] >> (8 * k)) & 0xFFu);
            const float d = (float)((c[2 % kTaps] >> (8 * k)) & 0xFFu), f = (float)((c[3 % kTaps] >> (8 * k)) & 0xFFu);
            if (SS == 2u) {
                const float top = __fmaf_rn(ax, __fsub_rn(b, a), a), bottom = __fmaf_rn(ax, __fsub_rn(f, d), d);
                out[k] = __fmul_rn(__fmaf_rn(ay, __fsub_rn(bottom, top), top), 1.0f / 255.f);
            } else {   // the neighbours at 1/8 each, the centre at 1/2
                const float wt = 0.125f;
                float s = __fmaf_rn(a, wt, 0.f);
                s = __fmaf_rn(b, wt, s);
                s = __fmaf_rn(d, wt, s);
                s = __fmaf_rn(f, wt, s);
                s = __fadd_rn(s, __fmul_rn((float)((c[4 % kTaps] >> (8 * k)) & 0xFFu), 0.5f));
                out[k] = __fmul_rn(s, 1.0f / 255.f);
            }
        }
        return f3(out[0], out[1], out[2]);
    }
};

template <uint32_t SS>
__device__ __forceinline__ F3 sample_as(const TexDev& t, float u, float v) {
    Lookup<SS> l;
    l.fetch(t, u, v);
    return l.colour();
}
__device__ __forceinline__ F3 sample_tex(const TexDev& t, float u, float v, uint32_t ss) {
    return ss == 2u ? sample_as<2>(t, u, v) : ss == 1u ? sample_as<1>(t, u, v) : sample_as<0>(t, u, v);
}

// Lambert + Phong over the scene lights (the build's extension, used when
// lights are set): per light the reference shader's terms with its constant
// light replaced -- L = the direction the light travels at P (a point
// light's from its position to P), irradiance E = intensity (/ squared
// distance for a point light, PointLight::GetBiradiance), diffuse +=
// diffuse * colour * max(0, dot(-N, L)) / pi * E, specular += specular *
// colour * clamp(dot(vd, reflect(L, N)), 0, 1)^(gloss * 25); then ambient +
// diffuse + specular and MaxToOne (CUDAROPs.cu:452-455), or the diffuse
// term alone without the specular and gloss maps (:459-462).
__device__ __forceinline__ F3 shade_lit(const LightDev* lights, uint32_t num_lights, F3 diffuse, F3 fn, F3 vd, F3 P, bool has_spec, F3 spec,
                                        F3 gloss) {
    F3 dacc = f3(0.f, 0.f, 0.f), sacc = f3(0.f, 0.f, 0.f);
    const F3 nfn = f3(-fn.x, -fn.y, -fn.z);
    const uint32_t nl = num_lights < kMaxLights ? num_lights : kMaxLights;
    for (uint32_t k = 0; k < nl; ++k) {
        const LightDev& lt = lights[k];
        F3 L;
        float E;
        if (lt.type == 1u) {
            const F3 d = f3(__fsub_rn(P.x, lt.vec[0]), __fsub_rn(P.y, lt.vec[1]), __fsub_rn(P.z, lt.vec[2]));
            E = __fdiv_rn(lt.intensity, dot3(d, d));
            L = normalize3(d);
        } else {
            L = f3(lt.vec[0], lt.vec[1], lt.vec[2]);
            E = lt.intensity;
        }
        float obs = dot3(nfn, L);
        obs = obs > 0.f ? obs : 0.f;
        obs = __fdiv_rn(obs, 3.14159265358979323846f);
        obs = __fmul_rn(obs, E);
        dacc = f3(__fmaf_rn(__fmul_rn(diffuse.x, lt.colour[0]), obs, dacc.x),
                  __fmaf_rn(__fmul_rn(diffuse.y, lt.colour[1]), obs, dacc.y),
                  __fmaf_rn(__fmul_rn(diffuse.z, lt.colour[2]), obs, dacc.z));
        if (has_spec) {
            const float s2 = __fmul_rn(2.f, dot3(L, fn));
            const F3 refl = f3(__fmaf_rn(fn.x, s2, -L.x), __fmaf_rn(fn.y, s2, -L.y), __fmaf_rn(fn.z, s2, -L.z));
            float ang = dot3(vd, refl);
            ang = ang < 0.f ? 0.f : (ang > 1.f ? 1.f : ang);
            ang = powf(ang, __fmul_rn(gloss.x, 25.f));
            sacc = f3(__fmaf_rn(__fmul_rn(spec.x, lt.colour[0]), ang, sacc.x),
                      __fmaf_rn(__fmul_rn(spec.y, lt.colour[1]), ang, sacc.y),
                      __fmaf_rn(__fmul_rn(spec.z, lt.colour[2]), ang, sacc.z));
        }
    }
    if (!has_spec) return dacc;
    F3 fc = f3(__fadd_rn(0.05f, dacc.x), __fadd_rn(0.05f, dacc.y), __fadd_rn(0.05f, dacc.z));
    fc = f3(__fadd_rn(fc.x, sacc.x), __fadd_rn(fc.y, sacc.y), __fadd_rn(fc.z, sacc.z));
    float mx = fc.y < fc.z ? fc.z : fc.y;
    mx = fc.x < mx ? mx : fc.x;
    if (mx > 1.f) {
        const float rev = __fdiv_rn(1.0f, mx);
        fc = f3(__fmul_rn(fc.x, rev), __fmul_rn(fc.y, rev), __fmul_rn(fc.z, rev));
    }
    return fc;
}

// RGBA::GetRGBAFromColour (RGBRaw.h:24-32): bytes B, G, R, 0.
__device__ __forceinline__ uint32_t rgba_from_colour(F3 c) {
    return cvt_u8(__fmul_rn(c.z, 255.f)) | (cvt_u8(__fmul_rn(c.y, 255.f)) << 8) | (cvt_u8(__fmul_rn(c.x, 255.f)) << 16);
}

// ShadePixelSafe (CUDAROPs.cu:411-470).
template <uint32_t SS>
__device__ __forceinline__ F3 shade_pixel_safe(const LightDev* lights, uint32_t num_lights, const MeshDev& m, float u,
                                               float v, F3 n, F3 tan, F3 vd, F3 P) {
    const F3 L = f3(0.577f, -0.577f, -0.577f);
    const bool has_spec = m.tex[1].px && m.tex[2].px && m.tex[3].px;
    Lookup<SS> ld, ln, ls, lg;
    ld.fetch(m.tex[0], u, v);
    if (m.tex[1].px) ln.fetch(m.tex[1], u, v);
    if (has_spec) {
        ls.fetch(m.tex[2], u, v);
        lg.fetch(m.tex[3], u, v);
    }
    const F3 diffuse = ld.colour();
    if (!m.tex[1].px) return diffuse;
    const F3 ns = ln.colour();
    const F3 cr = cross3(tan, n);
    const F3 bin = f3(-cr.x, -cr.y, -cr.z);
    const F3 fn0 = f3(__fmaf_rn(2.f, ns.x, -1.f), __fmaf_rn(2.f, ns.y, -1.f), __fmaf_rn(2.f, ns.z, -1.f));
    const F3 fn = f3(__fmaf_rn(n.x, fn0.z, __fmaf_rn(tan.x, fn0.x, __fmul_rn(bin.x, fn0.y))),
                     __fmaf_rn(n.y, fn0.z, __fmaf_rn(tan.y, fn0.x, __fmul_rn(bin.y, fn0.y))),
                     __fmaf_rn(n.z, fn0.z, __fmaf_rn(tan.z, fn0.x, __fmul_rn(bin.z, fn0.y))));
    if (num_lights) {
        const F3 zero = f3(0.f, 0.f, 0.f);
        const F3 spec = has_spec ? ls.colour() : zero;
        const F3 gloss = has_spec ? lg.colour() : zero;
        return shade_lit(lights, num_lights, diffuse, fn, vd, P, has_spec, spec, gloss);
    }
    float obs = dot3(f3(-fn.x, -fn.y, -fn.z), L);
    {   // ClampFast(obs, 0, obs) (CUDAROPs.cu:439) leaves negative values as they are
        const float c = obs < 0.f ? 0.f : obs;
        obs = c > obs ? obs : c;
    }
    obs = __fdiv_rn(obs, 3.14159265358979323846f);
    obs = __fmul_rn(obs, 7.0f);
    const F3 dcol = f3(__fmul_rn(diffuse.x, obs), __fmul_rn(diffuse.y, obs), __fmul_rn(diffuse.z, obs));
    if (!has_spec) return dcol;
    const F3 spec = ls.colour(), gloss = lg.colour();
    const float s2 = __fmul_rn(2.f, dot3(L, fn));
    const F3 refl = f3(__fmaf_rn(fn.x, s2, -L.x), __fmaf_rn(fn.y, s2, -L.y), __fmaf_rn(fn.z, s2, -L.z));
    float ang = dot3(vd, refl);
    ang = ang < 0.f ? 0.f : (ang > 1.f ? 1.f : ang);
    ang = powf(ang, __fmul_rn(gloss.x, 25.f));
    F3 fc = f3(__fadd_rn(0.05f, dcol.x), __fadd_rn(0.05f, dcol.y), __fadd_rn(0.05f, dcol.z));
    fc = f3(__fadd_rn(fc.x, __fmul_rn(spec.x, ang)), __fadd_rn(fc.y, __fmul_rn(spec.y, ang)),
            __fadd_rn(fc.z, __fmul_rn(spec.z, ang)));
    float mx = fc.y < fc.z ? fc.z : fc.y;   // MaxToOne (RGBColor.h:74-79)
    mx = fc.x < mx ? mx : fc.x;
    if (mx > 1.f) {
        const float rev = __fdiv_rn(1.0f, mx);
        fc = f3(__fmul_rn(fc.x, rev), __fmul_rn(fc.y, rev), __fmul_rn(fc.z, rev));
    }
    return fc;
}

// Colour of a fragment shaded from vertex colours (PBR view, no diffuse map):
// triangle `local` of mesh m, weights w.  The vertex colours are weighted by
// w / w_clip, not multiplied by the interpolated w (CUDAROPs.cu:379-380); of
// the vertex stage only each vertex's clip w and colour are needed, the same
// operations as in vertex_stage.
__device__ __forceinline__ uint32_t shade_flat(const FlatMesh& m, uint32_t local, const float w[3]) {
    uint32_t vid[3];
    tri_vertex_ids(m, local, vid);
    float ic[3];
    F3 col[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        F3 p;
        if (m.vertex_format == kVertexPos3Rgba8) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(m.vertices) + vid[k]);
            const uint32_t rgba = __float_as_uint(v.w);
            p = f3(v.x, v.y, v.z);
            col[k] = f3(over255(rgba & 0xFFu), over255((rgba >> 8) & 0xFFu), over255((rgba >> 16) & 0xFFu));
        } else {
            const float* b = reinterpret_cast<const float*>(m.vertices) + 14u * (size_t)vid[k];
            const float2 xy = __ldg(reinterpret_cast<const float2*>(b));
            const float2 gb = __ldg(reinterpret_cast<const float2*>(b + 12));
            p = f3(xy.x, xy.y, __ldg(b + 2));
            col[k] = f3(__ldg(b + 11), gb.x, gb.y);
        }
        const float cw = __fadd_rn(__fmaf_rn(m.w[2], p.z, __fmaf_rn(m.w[0], p.x, __fmul_rn(m.w[1], p.y))), m.w[3]);
        ic[k] = __frcp_rn(cw);   // 1 / cw, rounded as the division is
    }
#define GBR_CINTERP(a0, a1, a2) \
    __fmaf_rn(w[2], __fmul_rn((a2), ic[2]), __fmaf_rn(w[0], __fmul_rn((a0), ic[0]), __fmul_rn(w[1], __fmul_rn((a1), ic[1]))))
    const F3 c = f3(GBR_CINTERP(col[0].x, col[1].x, col[2].x), GBR_CINTERP(col[0].y, col[1].y, col[2].y),
                    GBR_CINTERP(col[0].z, col[1].z, col[2].z));
#undef GBR_CINTERP
    return rgba_from_colour(c);
}

// Remap(z, 0.985, 1) * 255 into the blue byte: the depth view.
__device__ __forceinline__ uint32_t shade_depth(float z) {
    const float rz = __fdiv_rn(__fsub_rn(z, 0.985f), __fsub_rn(1.f, 0.985f));
    return cvt_u8(__fmul_rn(rz, 255.f)) << 16;
}

// Colour of the fragment of primitive `prim` with weights w and depth z.
__device__ __forceinline__ uint32_t shade_fragment(const FrameDev& F, const MeshDev& m, const LightDev* lights,
                                                   uint32_t prim, const float w[3], float z) {
    if (F.vis == 1u) return shade_depth(z);
    if (F.vis == 0u && !m.tex[0].px) return shade_flat(flat_mesh(m), prim - m.prim_base, w);
    uint32_t vid[3];
    tri_vertex_ids(m, prim - m.prim_base, vid);
    const OVtx v0 = vertex_stage(m, F, vid[0]);
    const OVtx v1 = vertex_stage(m, F, vid[1]);
    const OVtx v2 = vertex_stage(m, F, vid[2]);
    const float i0 = __fdiv_rn(1.f, v0.pw), i1 = __fdiv_rn(1.f, v1.pw), i2 = __fdiv_rn(1.f, v2.pw);
    const float winterp = __fdiv_rn(1.f, __fmaf_rn(i2, w[2], __fmaf_rn(i0, w[0], __fmul_rn(i1, w[1]))));
#define GBR_INTERP(a0, a1, a2) \
    __fmaf_rn(w[2], __fmul_rn((a2), i2), __fmaf_rn(w[0], __fmul_rn((a0), i0), __fmul_rn(w[1], __fmul_rn((a1), i1))))
    F3 n = f3(GBR_INTERP(v0.n.x, v1.n.x, v2.n.x), GBR_INTERP(v0.n.y, v1.n.y, v2.n.y), GBR_INTERP(v0.n.z, v1.n.z, v2.n.z));
    n = f3(__fmul_rn(n.x, winterp), __fmul_rn(n.y, winterp), __fmul_rn(n.z, winterp));
    if (F.vis == 2u) return rgba_from_colour(n);
    const float u = __fmul_rn(GBR_INTERP(v0.u, v1.u, v2.u), winterp);
    const float vv = __fmul_rn(GBR_INTERP(v0.v, v1.v, v2.v), winterp);
    // tangent is not multiplied by the interpolated w (CUDAROPs.cu:371-372)
    const F3 tan = f3(GBR_INTERP(v0.tan.x, v1.tan.x, v2.tan.x), GBR_INTERP(v0.tan.y, v1.tan.y, v2.tan.y),
                      GBR_INTERP(v0.tan.z, v1.tan.z, v2.tan.z));
    const F3 vd = normalize3(f3(GBR_INTERP(v0.vd.x, v1.vd.x, v2.vd.x), GBR_INTERP(v0.vd.y, v1.vd.y, v2.vd.y),
                                GBR_INTERP(v0.vd.z, v1.vd.z, v2.vd.z)));
    F3 P = f3(0.f, 0.f, 0.f);
    if (F.num_lights)   // world position, perspective-correct like uv
        P = f3(__fmul_rn(GBR_INTERP(v0.wp.x, v1.wp.x, v2.wp.x), winterp),
               __fmul_rn(GBR_INTERP(v0.wp.y, v1.wp.y, v2.wp.y), winterp),
               __fmul_rn(GBR_INTERP(v0.wp.z, v1.wp.z, v2.wp.z), winterp));
#undef GBR_INTERP
    const uint32_t nl = F.num_lights;
    const F3 c = F.sample == 2u   ? shade_pixel_safe<2>(lights, nl, m, u, vv, n, tan, vd, P)
                 : F.sample == 1u ? shade_pixel_safe<1>(lights, nl, m, u, vv, n, tan, vd, P)
                                  : shade_pixel_safe<0>(lights, nl, m, u, vv, n, tan, vd, P);
    return rgba_from_colour(c);
}

}  // namespace gbr

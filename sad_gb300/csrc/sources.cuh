// sources.cuh -- where per-pixel kernels read site data from, and the per-candidate
// gradient algebra shared by the autograd adjoint and the fused training kernel.
#pragma once

#include "common.cuh"
#include "packed.cuh"

namespace sad {

// ---------------------------------------------------------------------------
// site sources: raw [N,10] sites (API calls) or prepared SiteGeom/SiteColor (trainer)
// ---------------------------------------------------------------------------
struct RawSites {
    const Site* s;
    __device__ __forceinline__ void load(uint32_t id, SiteGeom& g, float3& c) const {
        const float2* q = reinterpret_cast<const float2*>(s + id);
        float2 a = __ldg(q), b = __ldg(q + 1), cc = __ldg(q + 2), d = __ldg(q + 3), e = __ldg(q + 4);
        // a = (px, py), b = (log_tau, radius), cc = (r, g), d = (b, dx), e = (dy, log_aniso)
        g = make_geom(a.x, a.y, b.x, b.y, d.y, e.x, e.y);
        c = make_float3(cc.x, cc.y, d.x);
    }
    __device__ __forceinline__ float px(uint32_t id) const { return __ldg(&s[id].px); }
    __device__ __forceinline__ void prepare() {}
};

struct PreparedSites {
    const SiteGeom* g;
    const SiteColor* c;
    __device__ __forceinline__ void load(uint32_t id, SiteGeom& geom, float3& col) const {
        geom = load_geom(g, id);
        float4 v = __ldg(reinterpret_cast<const float4*>(c + id));
        col = make_float3(v.x, v.y, v.z);
    }
    __device__ __forceinline__ float px(uint32_t id) const { return __ldg(&g[id].px); }
    __device__ __forceinline__ void prepare() {}
};

// Prepares n raw sites in caller scratch of sad_site_scratch_bytes(n) bytes (render.cu).
PreparedSites prepare_in_scratch(const float* sites, uint32_t n, void* scratch, cudaStream_t st);

// 16-byte quantised sites (packed.cuh), decoded per candidate; an inactive site reads as
// position (-1, -1) so it is skipped like a pruned one (packedActive,
// backends/metal/shaders/sad_common.metal:85-87).  prepare() loads the ranges once per thread.
struct PackedSites {
    const uint4* p;
    const float* quant;  // device PackedQuant
    float dim_x, dim_y;  // W-1, H-1
    PackedQuant q;
    __device__ __forceinline__ void prepare() { q = load_packed_quant(quant); }
    __device__ __forceinline__ void load(uint32_t id, SiteGeom& g, float3& c) const {
        uint4 w = __ldg(p + id);
        Site s = decode_packed_site(w, q, dim_x, dim_y);
        if (!packed_active(w.x)) s.px = s.py = -1.0f;
        g = make_geom(s.px, s.py, s.log_tau, s.radius, s.dx, s.dy, s.log_aniso);
        c = make_float3(s.r, s.g, s.b);
    }
};

// Per-candidate parameter gradients for dL/dpred; out in site order.  clamp_l1 selects
// the fused kernel's l2 = 1 / max(l1, 1e-8) (gradients.cu:383) over 1 / l1
// (sad_bindings.cu:166).  Every operation is written with its rounding: left to the compiler,
// which of two products a sum fuses depends on the code around it, and a fit's sums would
// depend on which of the gradient kernel's loops a tile takes.
__device__ __forceinline__ void candidate_grads(const SiteGeom& g, float3 col, float ux, float uy,
                                                float inv_s2, float inv_scale, float w,
                                                float3 dLdp, float3 pred, bool clamp_l1,
                                                float (&o)[10]) {
    o[4] = __fmul_rn(w, dLdp.x);
    o[5] = __fmul_rn(w, dLdp.y);
    o[6] = __fmul_rn(w, dLdp.z);
    const float dlogit = __fmaf_rn(o[6], __fsub_rn(col.z, pred.z),
                                   __fmaf_rn(o[4], __fsub_rn(col.x, pred.x),
                                             __fmul_rn(o[5], __fsub_rn(col.y, pred.y))));
    const float tau = g.tau;
    const float dx = __fsub_rn(ux, g.px), dy = __fsub_rn(uy, g.py);
    const float diff2 = __fmaf_rn(dy, dy, __fmul_rn(dx, dx));
    const float proj = __fmaf_rn(g.dy, dy, __fmul_rn(g.dx, dx));
    const float proj2 = __fmul_rn(proj, proj);
    const float perp2 = fmaxf(__fsub_rn(diff2, proj2), 0.0f);
    const float l1 = g.l1;
    const float l2 = (clamp_l1 && !(l1 >= 1e-8f)) ? 1.0f / 1e-8f : g.l2;
    const float across = __fmul_rn(l2, perp2);
    const float d2s = fmaxf(__fmul_rn(__fmaf_rn(l1, proj2, across), inv_s2), 1e-8f);
    const float isq = rsqrtf(d2s);
    // sqrt(d2s) from the reciprocal root already at hand
    const float dm = __fmaf_rn(d2s, isq, -__fmul_rn(g.radius, inv_scale));
    const float axes = __fsub_rn(l1, l2);
    const float gdx = __fmaf_rn(l2, dx, __fmul_rn(__fmul_rn(axes, g.dx), proj));
    const float gdy = __fmaf_rn(l2, dy, __fmul_rn(__fmul_rn(axes, g.dy), proj));
    const float kpos = __fmul_rn(dlogit, __fmul_rn(__fmul_rn(tau, inv_s2), isq));
    o[0] = __fmul_rn(kpos, gdx);
    o[1] = __fmul_rn(kpos, gdy);
    o[2] = __fmul_rn(__fmul_rn(dlogit, -dm), tau);
    o[3] = __fmul_rn(__fmul_rn(dlogit, tau), inv_scale);
    const float dla = __fmul_rn(__fmaf_rn(l1, proj2, -across), inv_s2);
    const float kang = __fmul_rn(__fmul_rn(dlogit, -tau), __fmul_rn(0.5f, isq));
    const float kdir = __fmul_rn(__fmul_rn(__fmul_rn(2.0f, axes), proj), inv_s2);
    o[7] = __fmul_rn(kang, __fmul_rn(kdir, dx));
    o[8] = __fmul_rn(kang, __fmul_rn(kdir, dy));
    o[9] = __fmul_rn(kang, dla);
}

}  // namespace sad

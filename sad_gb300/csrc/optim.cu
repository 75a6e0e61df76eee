// optim.cu -- per-site optimisation: log-tau gradient diffusion, Adam, gradient clears.
//
// Trainer forms keep every iteration-dependent scalar on the device (DevState), so one
// captured CUDA graph per iteration kind is replayed for the whole fit:
//   * tau diffusion: lambda = 0.05 (0.1 + 0.9 iter / iters), the host formula of
//     backends/cuda/src/sad_cuda.cu:2339-2340, evaluated without contraction like an
//     x86 host build would;
//   * Adam: t = iter + 1 (sad_cuda.cu:2369-2380), fused with the gradient clear
//     (adam.cu:183-209) and with the refresh of the prepared SiteGeom/SiteColor records
//     the per-pixel kernels gather.
#include "accum.cuh"
#include "common.cuh"
#include "host_common.h"
#include "kernels.h"

namespace sad {

// ---------------------------------------------------------------------------
// tau diffusion (backends/cuda/src/tau_diffusion.cu:27-89)
// ---------------------------------------------------------------------------
template <class PosFn, class RawFn, class GinFn>
__device__ __forceinline__ float tau_diffuse_one(uint32_t i, const uint4* __restrict__ c0,
                                                 const uint4* __restrict__ c1, PosFn pos,
                                                 RawFn raw, GinFn gin, uint32_t n, float lambda,
                                                 int w, int h, int ds) {
    float2 sp = pos(i);
    if (lambda <= 0.0f || sp.x < 0.0f) return gin(i);
    float inv = 1.0f / fmaxf(static_cast<float>(ds), 1.0f);
    int px = clampi(static_cast<int>(sp.x * inv + 0.5f), 0, w - 1);
    int py = clampi(static_cast<int>(sp.y * inv + 0.5f), 0, h - 1);
    int p = py * w + px;
    uint4 a = __ldg(c0 + p), b = __ldg(c1 + p);
    uint32_t ids[kCand] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    float sum = 0.0f;
    uint32_t cnt = 0;
#pragma unroll
    for (int k = 0; k < kCand; ++k) {
        uint32_t m = ids[k];
        if (m >= n || m == i) continue;
        bool seen = false;
#pragma unroll
        for (int j = 0; j < k; ++j) seen |= ids[j] == m;
        if (seen) continue;
        if (pos(m).x < 0.0f) continue;
        sum += gin(m);
        cnt += 1;
    }
    float diag = 1.0f + lambda * static_cast<float>(cnt);
    return (raw(i) + lambda * sum) / diag;
}

__global__ void tau_diffuse_raw_kernel(const uint4* __restrict__ c0, const uint4* __restrict__ c1,
                                       const Site* __restrict__ sites, const float* __restrict__ raw,
                                       const float* __restrict__ gin, float* __restrict__ gout,
                                       uint32_t n, float lambda, int w, int h, int ds) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    auto pos = [sites](uint32_t k) { return make_float2(__ldg(&sites[k].px), __ldg(&sites[k].py)); };
    auto rawf = [raw](uint32_t k) { return raw[k]; };
    auto ginf = [gin](uint32_t k) { return gin[k]; };
    gout[i] = tau_diffuse_one(i, c0, c1, pos, rawf, ginf, n, lambda, w, h, ds);
}

void launch_tau_diffuse_raw(const uint32_t* c0, const uint32_t* c1, const Site* sites,
                            const float* raw, const float* gin, float* gout, uint32_t n,
                            float lambda, int w, int h, int ds, cudaStream_t st) {
    if (n == 0) return;
    tau_diffuse_raw_kernel<<<blocks_for(n, 256), 256, 0, st>>>(
        reinterpret_cast<const uint4*>(c0), reinterpret_cast<const uint4*>(c1), sites, raw, gin,
        gout, n, lambda, w, h, ds);
    note_launches(1);
}

__device__ __forceinline__ float tau_lambda(uint32_t iter, int iterations) {
    float blend = __fdiv_rn(static_cast<float>(iter), static_cast<float>(max(1, iterations)));
    return __fmul_rn(0.05f, __fadd_rn(0.1f, __fmul_rn(0.9f, blend)));
}

// Trainer form.  The four Jacobi passes of an iteration share one candidate field and one
// set of positions, so the first pass records each active site's neighbour list (the
// distinct active candidates at its texel, in candidate order) and the raw gradient as a
// float; the middle passes read the list; the last pass runs inside the Adam kernel.
// Every pass walks the compacted list of active sites (state->n_alive entries): an
// inactive site's diffused value is never read (a neighbour must be active, and Adam
// skips inactive sites).  by_position: some sites have position.x NaN, which makes them
// neither active nor, to the gradient kernel and the candidate passes, inactive.
struct TauLists {
    uint4* nbr;            // [n][2] neighbour ids, kEmpty-padded
    float* raw;            // [n] raw log-tau gradient (float)
    const uint32_t* alive; // the compacted active list
};

__device__ __forceinline__ void tau_first_one(const uint4* __restrict__ c0, const uint4* __restrict__ c1,
                                              const SiteGeom* __restrict__ geom,
                                              const long long* __restrict__ fix12, const TauLists& tl,
                                              float* __restrict__ gout, uint32_t n, uint32_t i,
                                              float lambda, int w, int h, int ds, bool by_position);

__global__ void tau_first_pass_kernel(const uint4* __restrict__ c0, const uint4* __restrict__ c1,
                                      const SiteGeom* __restrict__ geom,
                                      const long long* __restrict__ fix12, TauLists tl,
                                      float* __restrict__ gout, uint32_t n,
                                      const DevState* __restrict__ state, int iterations, int w,
                                      int h, int ds, bool by_position) {
    pdl_wait();
    const uint32_t n_alive = state->n_alive;
    const float lambda = tau_lambda(state->iter, iterations);
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n_alive; j += gridDim.x * blockDim.x) {
        const uint32_t i = tl.alive[j];
        tau_first_one(c0, c1, geom, fix12, tl, gout, n, i, lambda, w, h, ds, by_position);
    }
}

__device__ __forceinline__ void tau_first_one(const uint4* __restrict__ c0, const uint4* __restrict__ c1,
                                              const SiteGeom* __restrict__ geom,
                                              const long long* __restrict__ fix12, const TauLists& tl,
                                              float* __restrict__ gout, uint32_t n, uint32_t i,
                                              float lambda, int w, int h, int ds, bool by_position) {
    float2 sp = __ldg(reinterpret_cast<const float2*>(geom + i));
    const float r = from_fix(fix12[static_cast<size_t>(i) * 12 + kTauWord]);
    tl.raw[i] = r;
    float inv = 1.0f / fmaxf(static_cast<float>(ds), 1.0f);
    int px = clampi(static_cast<int>(sp.x * inv + 0.5f), 0, w - 1);
    int py = clampi(static_cast<int>(sp.y * inv + 0.5f), 0, h - 1);
    int p = py * w + px;
    uint4 a = __ldg(c0 + p), b = __ldg(c1 + p);
    uint32_t ids[kCand] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    // every candidate's raw gradient is fetched before any is used, so the gathers overlap
    // instead of forming a chain of dependent loads; an inactive site's word says so (with its
    // position gathered too, the pass over a 6-image batch's 768,000 sites took 66 us).  The
    // word alone does not: the sum of an active site can come to it (a NaN or infinite term
    // does), so the position decides for the few that carry it.
    long long cfix[kCand];
#pragma unroll
    for (int k = 0; k < kCand; ++k) {
        const uint32_t m = ids[k];
        cfix[k] = m < n && m != i ? fix12[static_cast<size_t>(m) * 12 + kTauWord] : kInactiveWord;
    }
    uint32_t list[kCand];
    float sum = 0.0f;
    uint32_t cnt = 0;
#pragma unroll
    for (int k = 0; k < kCand; ++k) {
        list[k] = kEmpty;
        uint32_t m = ids[k];
        bool take = cfix[k] != kInactiveWord;
        if (by_position || !take) take = m < n && m != i && __ldg(&geom[m].px) >= 0.0f;
#pragma unroll
        for (int j = 0; j < k; ++j) take &= ids[j] != m;
        if (take) {
            sum += from_fix(cfix[k]);
            list[k] = m;
            cnt += 1;
        }
    }
    tl.nbr[2 * i] = make_uint4(list[0], list[1], list[2], list[3]);
    tl.nbr[2 * i + 1] = make_uint4(list[4], list[5], list[6], list[7]);
    if (!(lambda > 0.0f)) {
        gout[i] = r;
        return;
    }
    gout[i] = (r + lambda * sum) / (1.0f + lambda * static_cast<float>(cnt));
}

// One Jacobi pass of an active site from its recorded neighbour list (sum in candidate
// order, as the first pass and the reference's kernel); gin(i): the last pass's value.
template <class Gin>
__device__ __forceinline__ float tau_list_pass(const TauLists& tl, Gin gin, uint32_t i, float lambda) {
    const float r = tl.raw[i];
    if (!(lambda > 0.0f)) return gin(i);
    uint4 a = tl.nbr[2 * i], b = tl.nbr[2 * i + 1];
    uint32_t ids[kCand] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    float v[kCand];
#pragma unroll
    for (int k = 0; k < kCand; ++k) v[k] = ids[k] == kEmpty ? 0.0f : gin(ids[k]);  // gathers overlap
    float sum = 0.0f;
    uint32_t cnt = 0;
#pragma unroll
    for (int k = 0; k < kCand; ++k) {
        if (ids[k] == kEmpty) continue;
        sum += v[k];
        cnt += 1;
    }
    return (r + lambda * sum) / (1.0f + lambda * static_cast<float>(cnt));
}

__global__ void tau_list_pass_kernel(TauLists tl, const float* __restrict__ gin,
                                     float* __restrict__ gout, const DevState* __restrict__ state,
                                     int iterations) {
    pdl_wait();
    const uint32_t n_alive = state->n_alive;
    const float lambda = tau_lambda(state->iter, iterations);
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n_alive; j += gridDim.x * blockDim.x) {
        const uint32_t i = tl.alive[j];
        gout[i] = tau_list_pass(tl, [gin](uint32_t k) { return gin[k]; }, i, lambda);
    }
}

void launch_tau_first_pass(const uint32_t* c0, const uint32_t* c1, const SiteGeom* geom,
                           const long long* fix12, uint32_t* nbr, float* raw, const uint32_t* alive,
                           float* gout, uint32_t n, uint32_t max_alive, const DevState* state,
                           int iterations, int w, int h, int ds, bool by_position, cudaStream_t st) {
    if (max_alive == 0) return;
    TauLists tl{reinterpret_cast<uint4*>(nbr), raw, alive};
    launch_pdl(tau_first_pass_kernel, dim3(blocks_for(max_alive, 256)), dim3(256), 0, st,
               reinterpret_cast<const uint4*>(c0), reinterpret_cast<const uint4*>(c1), geom, fix12, tl, gout, n,
               state, iterations, w, h, ds, by_position);
    note_launches(1);
}

void launch_tau_list_pass(const uint32_t* nbr, const float* raw, const uint32_t* alive,
                          const float* gin, float* gout, uint32_t max_alive, const DevState* state,
                          int iterations, cudaStream_t st) {
    if (max_alive == 0) return;
    TauLists tl{reinterpret_cast<uint4*>(const_cast<uint32_t*>(nbr)), const_cast<float*>(raw), alive};
    launch_pdl(tau_list_pass_kernel, dim3(blocks_for(max_alive, 256)), dim3(256), 0, st, tl, gin, gout, state,
               iterations);
    note_launches(1);
}

// ---------------------------------------------------------------------------
// Adam (backends/cuda/src/adam.cu:5-180)
// ---------------------------------------------------------------------------
struct AdamSlots {  // the 20-float per-site state
    float v[20];
};

__device__ __forceinline__ void adam_load(const float* __restrict__ a, uint32_t i, AdamSlots& s) {
    const float4* q = reinterpret_cast<const float4*>(a + static_cast<size_t>(i) * 20);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        float4 t = q[k];
        s.v[4 * k] = t.x; s.v[4 * k + 1] = t.y; s.v[4 * k + 2] = t.z; s.v[4 * k + 3] = t.w;
    }
}

__device__ __forceinline__ void adam_store(float* __restrict__ a, uint32_t i, const AdamSlots& s) {
    float4* q = reinterpret_cast<float4*>(a + static_cast<size_t>(i) * 20);
#pragma unroll
    for (int k = 0; k < 5; ++k)
        q[k] = make_float4(s.v[4 * k], s.v[4 * k + 1], s.v[4 * k + 2], s.v[4 * k + 3]);
}

// One Adam step of one active site.  g[] = the 10 normalised gradients in site order.
__device__ __forceinline__ void adam_site(Site& s, AdamSlots& a, const float (&g)[10],
                                          const AdamHyper& hp, float c1, float c2, int w, int h) {
    const float b1 = hp.beta1, b2 = hp.beta2, eps = hp.eps;
    // position: isotropic Adam
    a.v[0] = b1 * a.v[0] + (1.0f - b1) * g[0];
    a.v[1] = b1 * a.v[1] + (1.0f - b1) * g[1];
    float g2p = g[0] * g[0] + g[1] * g[1];
    a.v[2] = b2 * a.v[2] + (1.0f - b2) * g2p;
    {
        float mh0 = a.v[0] * c1, mh1 = a.v[1] * c1;
        float vh = a.v[2] * c2;
        float idn = 1.0f / (sqrtf(vh) + eps);
        float st0 = hp.lr_pos * mh0 * idn, st1 = hp.lr_pos * mh1 * idn;
        s.px -= st0;
        s.py -= st1;
        s.px = clampf(s.px, 0.0f, static_cast<float>(w - 1));
        s.py = clampf(s.py, 0.0f, static_cast<float>(h - 1));
    }
    // log_tau
    a.v[3] = b1 * a.v[3] + (1.0f - b1) * g[2];
    a.v[4] = b2 * a.v[4] + (1.0f - b2) * (g[2] * g[2]);
    s.log_tau -= hp.lr_tau * (a.v[3] * c1) / (sqrtf(a.v[4] * c2) + eps);
    // radius
    a.v[5] = b1 * a.v[5] + (1.0f - b1) * g[3];
    a.v[6] = b2 * a.v[6] + (1.0f - b2) * (g[3] * g[3]);
    s.radius -= hp.lr_radius * (a.v[5] * c1) / (sqrtf(a.v[6] * c2) + eps);
    s.radius = clampf(s.radius, 1.0f, 512.0f);
    // colour, per channel
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        a.v[7 + c] = b1 * a.v[7 + c] + (1.0f - b1) * g[4 + c];
        a.v[10 + c] = b2 * a.v[10 + c] + (1.0f - b2) * (g[4 + c] * g[4 + c]);
    }
    float st_r = hp.lr_color * (a.v[7] * c1) / (sqrtf(a.v[10] * c2) + eps);
    float st_g = hp.lr_color * (a.v[8] * c1) / (sqrtf(a.v[11] * c2) + eps);
    float st_b = hp.lr_color * (a.v[9] * c1) / (sqrtf(a.v[12] * c2) + eps);
    s.r = clampf(s.r - st_r, 0.0f, 1.0f);
    s.g = clampf(s.g - st_g, 0.0f, 1.0f);
    s.b = clampf(s.b - st_b, 0.0f, 1.0f);
    // direction: tangent-space isotropic Adam, renormalised
    {
        float dx = s.dx, dy = s.dy;
        float gd = g[7] * dx + g[8] * dy;
        float gtx = g[7] - dx * gd, gty = g[8] - dy * gd;
        a.v[13] = b1 * a.v[13] + (1.0f - b1) * gtx;
        a.v[14] = b1 * a.v[14] + (1.0f - b1) * gty;
        float g2d = gtx * gtx + gty * gty;
        a.v[15] = b2 * a.v[15] + (1.0f - b2) * g2d;
        float mh0 = a.v[13] * c1, mh1 = a.v[14] * c1;
        float vh = a.v[15] * c2;
        float idn = 1.0f / (sqrtf(vh) + eps);
        float nx = dx - hp.lr_dir * mh0 * idn, ny = dy - hp.lr_dir * mh1 * idn;
        float l2 = nx * nx + ny * ny;
        if (l2 < 1e-12f) {
            nx = 1.0f;
            ny = 0.0f;
        } else {
            float il = rsqrtf(l2);
            nx *= il;
            ny *= il;
        }
        s.dx = nx;
        s.dy = ny;
    }
    // log_aniso
    a.v[16] = b1 * a.v[16] + (1.0f - b1) * g[9];
    a.v[17] = b2 * a.v[17] + (1.0f - b2) * (g[9] * g[9]);
    s.log_aniso -= hp.lr_aniso * (a.v[16] * c1) / (sqrtf(a.v[17] * c2) + eps);
    s.log_aniso = clampf(s.log_aniso, -4.0f, 4.0f);
}

__device__ __forceinline__ Site site_load(const Site* __restrict__ sites, uint32_t i) {
    const float2* q = reinterpret_cast<const float2*>(sites + i);
    float2 a = q[0], b = q[1], c = q[2], d = q[3], e = q[4];
    Site s;
    s.px = a.x; s.py = a.y; s.log_tau = b.x; s.radius = b.y; s.r = c.x; s.g = c.y;
    s.b = d.x; s.dx = d.y; s.dy = e.x; s.log_aniso = e.y;
    return s;
}

__device__ __forceinline__ void site_store(Site* __restrict__ sites, uint32_t i, const Site& s) {
    float2* q = reinterpret_cast<float2*>(sites + i);
    q[0] = make_float2(s.px, s.py);
    q[1] = make_float2(s.log_tau, s.radius);
    q[2] = make_float2(s.r, s.g);
    q[3] = make_float2(s.b, s.dx);
    q[4] = make_float2(s.dy, s.log_aniso);
}

struct SoaGrads {
    const float* g[10];
};

__global__ void adam_soa_kernel(Site* __restrict__ sites, float* __restrict__ adam, SoaGrads gr,
                                AdamHyper hp, uint32_t t, uint32_t n, int w, int h) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float norm = 1.0f / static_cast<float>(w * h);
    float g[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) g[k] = gr.g[k][i] * norm;
    Site s = site_load(sites, i);
    if (s.px < 0.0f) return;
    float tt = static_cast<float>(t);
    float c1 = 1.0f / (1.0f - powf(hp.beta1, tt));
    float c2 = 1.0f / (1.0f - powf(hp.beta2, tt));
    AdamSlots a;
    adam_load(adam, i, a);
    adam_site(s, a, g, hp, c1, c2, w, h);
    adam_store(adam, i, a);
    site_store(sites, i, s);
}

void launch_adam_soa(Site* sites, float* adam, const float* const g[10], const AdamHyper& hp,
                     uint32_t t, uint32_t n, int w, int h, cudaStream_t st) {
    if (n == 0) return;
    SoaGrads gr;
    for (int k = 0; k < 10; ++k) gr.g[k] = g[k];
    adam_soa_kernel<<<blocks_for(n, 256), 256, 0, st>>>(sites, adam, gr, hp, t, n, w, h);
    note_launches(1);
}

// Trainer form: the last tau Jacobi pass, then Adam on the fixed-point gradient records,
// which are consumed and cleared (slots 0-9; slots 10-11, the removal delta, belong to the
// prune step), then the refreshed SiteGeom / SiteColor records.  Inactive sites carry no
// gradient and are left untouched.
//
// A warp takes 32 sites of the active list.  Their rows (80 bytes of Adam state, 80 of a
// gradient record, 40 of the site) come and go through shared memory in chunks of a fifth of
// a row, neighbouring lanes neighbouring chunks, so that an instruction touches a few lines
// instead of one per lane; the copies in run while the tau pass gathers.  Bound by latency and
// the gathers.  (One row per lane kept the load queue full at 9% issue and 30% of L2's rate.)
constexpr int kAdamThreads = 128;

struct AdamStage {  // of one warp
    float4 adam[32][5];
    longlong2 grads[32][5];
    float2 site[32][5];
};

__device__ __forceinline__ void copy_async16(void* shared, const void* global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(shared))),
                 "l"(global)
                 : "memory");
}
__device__ __forceinline__ void copy_async8(void* shared, const void* global) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(shared))),
                 "l"(global)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The iteration's scalars.
struct StepScalars {
    float lambda, c1, c2;
};
__device__ __forceinline__ StepScalars step_scalars(const DevState* state, int iterations) {
    return StepScalars{tau_lambda(state->iter, iterations), state->adam_c1, state->adam_c2};
}

// All lanes of the warp; i: the lane's site, kEmpty for none; tau_gin(i): the third tau pass's
// value.
template <class Gin>
__device__ __forceinline__ void adam_train_warp(Site* __restrict__ sites, float* __restrict__ adam,
                                                long long* __restrict__ fix12, const TauLists& tl, Gin tau_gin,
                                                SiteGeom* __restrict__ geom, SiteColor* __restrict__ color,
                                                const AdamHyper& hp, const StepScalars& step, int w, int h,
                                                uint32_t i, AdamStage& stage) {
    const uint32_t lane = lane_id();
    float4* const adam_rows = &stage.adam[0][0];
    longlong2* const grad_rows = &stage.grads[0][0];
    float2* const site_rows = &stage.site[0][0];
    __syncwarp();  // the last sites' chunks are out
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const uint32_t c = lane + 32 * j, part = c % 5;
        const uint32_t id = __shfl_sync(0xffffffffu, i, c / 5);
        if (id == kEmpty) continue;
        copy_async16(grad_rows + c, reinterpret_cast<const longlong2*>(fix12 + static_cast<size_t>(id) * 12) + part);
        copy_async16(adam_rows + c, reinterpret_cast<const float4*>(adam + static_cast<size_t>(id) * 20) + part);
        copy_async8(site_rows + c, reinterpret_cast<const float2*>(sites + id) + part);
    }
    float tau_g = 0.0f;
    if (i != kEmpty) tau_g = tau_list_pass(tl, tau_gin, i, step.lambda);
    copy_async_wait();
    __syncwarp();
    if (i != kEmpty) {
        const float norm = 1.0f / static_cast<float>(w * h);
        longlong2 q[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) q[k] = stage.grads[lane][k];
        float g[10] = {from_fix(q[0].x) * norm, from_fix(q[0].y) * norm, tau_g * norm,
                       from_fix(q[1].y) * norm, from_fix(q[2].x) * norm, from_fix(q[2].y) * norm,
                       from_fix(q[3].x) * norm, from_fix(q[3].y) * norm, from_fix(q[4].x) * norm,
                       from_fix(q[4].y) * norm};
        Site s = site_load(reinterpret_cast<const Site*>(site_rows), lane);
        AdamSlots a;
        adam_load(reinterpret_cast<const float*>(adam_rows), lane, a);
        adam_site(s, a, g, hp, step.c1, step.c2, w, h);
        adam_store(reinterpret_cast<float*>(adam_rows), lane, a);
        site_store(reinterpret_cast<Site*>(site_rows), lane, s);
        store_geom(geom, i, make_geom(s.px, s.py, s.log_tau, s.radius, s.dx, s.dy, s.log_aniso));
        reinterpret_cast<float4*>(color)[i] = make_float4(s.r, s.g, s.b, 0.0f);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const uint32_t c = lane + 32 * j, part = c % 5;
        const uint32_t id = __shfl_sync(0xffffffffu, i, c / 5);
        if (id == kEmpty) continue;
        reinterpret_cast<longlong2*>(fix12 + static_cast<size_t>(id) * 12)[part] = make_longlong2(0, 0);
        reinterpret_cast<float4*>(adam + static_cast<size_t>(id) * 20)[part] = adam_rows[c];
        reinterpret_cast<float2*>(sites + id)[part] = site_rows[c];
    }
}

__global__ void __launch_bounds__(kAdamThreads)
    adam_train_kernel(Site* __restrict__ sites, float* __restrict__ adam, long long* __restrict__ fix12, TauLists tl,
                      const float* __restrict__ tau_gin, SiteGeom* __restrict__ geom, SiteColor* __restrict__ color,
                      AdamHyper hp, const DevState* __restrict__ state, int iterations, int w, int h) {
    __shared__ AdamStage stage[kAdamThreads / 32];
    pdl_wait();
    const uint32_t n_alive = state->n_alive;
    const StepScalars step = step_scalars(state, iterations);
    // whole warps: j differs by the lane only
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; (j & ~31u) < n_alive; j += gridDim.x * blockDim.x)
        adam_train_warp(sites, adam, fix12, tl, [tau_gin](uint32_t k) { return tau_gin[k]; }, geom, color, hp, step,
                        w, h, j < n_alive ? tl.alive[j] : kEmpty, stage[threadIdx.x / 32]);
}

void launch_adam_train(Site* sites, float* adam, long long* fix12, const uint32_t* nbr,
                       const float* raw, const uint32_t* alive, const float* tau_gin,
                       SiteGeom* geom, SiteColor* color, const AdamHyper& hp,
                       const DevState* state, int iterations, uint32_t max_alive, int w, int h,
                       cudaStream_t st) {
    if (max_alive == 0) return;
    TauLists tl{reinterpret_cast<uint4*>(const_cast<uint32_t*>(nbr)), const_cast<float*>(raw), alive};
    launch_pdl(adam_train_kernel, dim3(blocks_for(max_alive, kAdamThreads)), dim3(kAdamThreads), 0, st, sites, adam,
               fix12, tl, tau_gin, geom, color, hp, state, iterations, w, h);
    note_launches(1);
}

// ---------------------------------------------------------------------------
// clears and the iteration counter
// ---------------------------------------------------------------------------
__global__ void clear10_kernel(SoaGrads g, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int k = 0; k < 10; ++k) const_cast<float*>(g.g[k])[i] = 0.0f;
}

__device__ __forceinline__ void set_bias_corrections(DevState* state, float beta1, float beta2) {
    float tt = static_cast<float>(state->iter + 1u);  // Adam step t = iter + 1
    state->adam_c1 = 1.0f / (1.0f - powf(beta1, tt));
    state->adam_c2 = 1.0f / (1.0f - powf(beta2, tt));
}

__global__ void reset_state_kernel(DevState* state, float beta1, float beta2) {
    state->iter = 0u;
    state->vpt_pass = 0u;
    state->wide_far_refs = kWideFarRefs;
    set_bias_corrections(state, beta1, beta2);
}

__global__ void advance_state_kernel(DevState* state, uint32_t vpt_passes, float beta1, float beta2) {
    pdl_wait();
    state->iter += 1u;
    state->vpt_pass += vpt_passes;
    set_bias_corrections(state, beta1, beta2);
}

void launch_reset_state(DevState* state, float beta1, float beta2, cudaStream_t st) {
    reset_state_kernel<<<1, 1, 0, st>>>(state, beta1, beta2);
    note_launches(1);
}

__global__ void set_wide_far_refs_kernel(DevState* state, int value) { state->wide_far_refs = value; }

void launch_set_wide_far_refs(DevState* state, int value, cudaStream_t st) {
    set_wide_far_refs_kernel<<<1, 1, 0, st>>>(state, value);
    note_launches(1);
}

// The per-site work of an iteration in one launch, for fits of at most kChainSites sites: the
// three tau passes and Adam, a cluster barrier between them instead of a launch, and the state
// advance.  One cluster of kChainBlocks blocks (a barrier of which costs far less than a launch
// boundary); the passes exchange their values through L2.
constexpr int kChainBlocks = 16;
constexpr int kChainThreads = 256;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kChainThreads)
    site_chain_kernel(const uint4* __restrict__ c0, const uint4* __restrict__ c1, Site* sites, float* adam,
                      long long* fix12, TauLists tl, float* tau_a, float* tau_b, SiteGeom* geom, SiteColor* color,
                      AdamHyper hp, DevState* state, int iterations, uint32_t n, int cw, int ch, int ds, int w, int h,
                      bool by_position, bool advance, uint32_t vpt_passes) {
    extern __shared__ __align__(16) unsigned char sad_chain_smem[];
    pdl_wait();
    const uint32_t n_alive = state->n_alive;
    const StepScalars step = step_scalars(state, iterations);
    const uint32_t first = blockIdx.x * kChainThreads + threadIdx.x, stride = kChainBlocks * kChainThreads;
    for (uint32_t j = first; j < n_alive; j += stride)
        tau_first_one(c0, c1, geom, fix12, tl, tau_a, n, tl.alive[j], step.lambda, cw, ch, ds,
                      by_position);
    cluster_barrier();
    if (advance && first == 0) {  // every block has read the state
        state->iter += 1u;
        state->vpt_pass += vpt_passes;
        set_bias_corrections(state, hp.beta1, hp.beta2);
    }
    const float* gin = tau_a;
    float* gout = tau_b;
    for (int pass = 0; pass < 2; ++pass) {
        for (uint32_t j = first; j < n_alive; j += stride) {
            const uint32_t i = tl.alive[j];
            gout[i] = tau_list_pass(tl, [gin](uint32_t k) { return __ldcg(gin + k); }, i, step.lambda);
        }
        cluster_barrier();
        gin = tau_b;
        gout = tau_a;
    }
    AdamStage& stage = reinterpret_cast<AdamStage*>(sad_chain_smem)[threadIdx.x / 32];
    for (uint32_t j = first; (j & ~31u) < n_alive; j += stride)
        adam_train_warp(sites, adam, fix12, tl, [tau_a](uint32_t k) { return __ldcg(tau_a + k); }, geom, color, hp,
                        step, w, h, j < n_alive ? tl.alive[j] : kEmpty, stage);
}

cudaError_t prepare_site_chain() {
    cudaError_t e = cudaFuncSetAttribute(site_chain_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(site_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kChainThreads / 32 * sizeof(AdamStage)));
    return e;
}

void launch_site_chain(const uint32_t* c0, const uint32_t* c1, Site* sites, float* adam, long long* fix12,
                       uint32_t* nbr, float* raw, const uint32_t* alive, float* tau_a, float* tau_b, SiteGeom* geom,
                       SiteColor* color, const AdamHyper& hp, DevState* state, int iterations, uint32_t n, int cw,
                       int ch, int ds, int w, int h, bool by_position, bool advance, uint32_t vpt_passes,
                       cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kChainBlocks);
    cfg.blockDim = dim3(kChainThreads);
    cfg.dynamicSmemBytes = kChainThreads / 32 * sizeof(AdamStage);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = kChainBlocks;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    TauLists tl{reinterpret_cast<uint4*>(nbr), raw, alive};
    cudaLaunchKernelEx(&cfg, site_chain_kernel, reinterpret_cast<const uint4*>(c0), reinterpret_cast<const uint4*>(c1),
                       sites, adam, fix12, tl, tau_a, tau_b, geom, color, hp, state, iterations, n, cw, ch, ds, w, h,
                       by_position, advance, vpt_passes);
    note_launches(1);
}

void launch_advance_state(DevState* state, uint32_t vpt_passes, float beta1, float beta2,
                          cudaStream_t st) {
    launch_pdl(advance_state_kernel, dim3(1), dim3(1), 0, st, state, vpt_passes, beta1, beta2);
    note_launches(1);
}

// ---------------------------------------------------------------------------
// batched forms: every image of a batch in one launch, over the flat active list
// ---------------------------------------------------------------------------
__global__ void batch_site_prefix_kernel(const SiteBatchItem* __restrict__ items, uint32_t n_items,
                                         uint32_t* __restrict__ prefix) {
    pdl_wait();
    if (threadIdx.x != 0) return;
    uint32_t run = 0;
    for (uint32_t i = 0; i < n_items; ++i) {
        prefix[i] = run;
        run += items[i].state->n_alive;
    }
    prefix[n_items] = run;
}

void launch_batch_site_prefix(const SiteBatchItem* items, uint32_t n_items, uint32_t* site_prefix, cudaStream_t st) {
    launch_pdl(batch_site_prefix_kernel, dim3(1), dim3(32), 0, st, items, n_items, site_prefix);
    note_launches(1);
}

__global__ void __launch_bounds__(256) tau_first_batch_kernel(const SiteBatchItem* __restrict__ items,
                                                              const uint32_t* __restrict__ prefix,
                                                              uint32_t n_items, int field, int iterations) {
    pdl_wait();
    __shared__ uint32_t s_prefix[kMaxBatchItems + 1];
    const uint32_t total = load_site_prefix(s_prefix, prefix, n_items);
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const uint32_t k = batch_item_of(s_prefix, n_items, g);
        const SiteBatchItem& it = items[k];
        TauLists tl{reinterpret_cast<uint4*>(it.tau_nbr), it.tau_raw, it.alive};
        const uint32_t i = it.alive[g - s_prefix[k]];
        tau_first_one(reinterpret_cast<const uint4*>(it.cand0[field]), reinterpret_cast<const uint4*>(it.cand1[field]),
                      it.geom, it.grads, tl, it.tau_a, it.n, i, tau_lambda(it.state->iter, iterations), it.cw,
                      it.ch, it.ds, false);
    }
}

__global__ void __launch_bounds__(256) tau_list_batch_kernel(const SiteBatchItem* __restrict__ items,
                                                             const uint32_t* __restrict__ prefix,
                                                             uint32_t n_items, int a_to_b, int iterations) {
    pdl_wait();
    __shared__ uint32_t s_prefix[kMaxBatchItems + 1];
    const uint32_t total = load_site_prefix(s_prefix, prefix, n_items);
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const uint32_t k = batch_item_of(s_prefix, n_items, g);
        const SiteBatchItem& it = items[k];
        TauLists tl{reinterpret_cast<uint4*>(it.tau_nbr), it.tau_raw, it.alive};
        const uint32_t i = it.alive[g - s_prefix[k]];
        const float* gin = a_to_b ? it.tau_a : it.tau_b;
        float* gout = a_to_b ? it.tau_b : it.tau_a;
        gout[i] = tau_list_pass(tl, [gin](uint32_t k) { return gin[k]; }, i, tau_lambda(it.state->iter, iterations));
    }
}

__global__ void __launch_bounds__(kAdamThreads) adam_batch_kernel(const SiteBatchItem* __restrict__ items,
                                                                  const uint32_t* __restrict__ prefix,
                                                                  uint32_t n_items, AdamHyper hp, int iterations) {
    pdl_wait();
    __shared__ uint32_t s_prefix[kMaxBatchItems + 1];
    __shared__ AdamStage stage[kAdamThreads / 32];
    const uint32_t total = load_site_prefix(s_prefix, prefix, n_items);
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; (g & ~31u) < total; g += gridDim.x * blockDim.x) {
        // one image after the other: a warp's sites are mostly one image's
        const uint32_t mine = g < total ? batch_item_of(s_prefix, n_items, g) : kEmpty;
        uint32_t todo = __ballot_sync(0xffffffffu, mine != kEmpty);
        while (todo != 0u) {
            const uint32_t k = __shfl_sync(0xffffffffu, mine, __ffs(todo) - 1);
            const SiteBatchItem& it = items[k];
            TauLists tl{reinterpret_cast<uint4*>(it.tau_nbr), it.tau_raw, it.alive};
            const float* gin = it.tau_a;
            adam_train_warp(it.sites, it.adam, it.grads, tl, [gin](uint32_t m) { return gin[m]; }, it.geom, it.color,
                            hp, step_scalars(it.state, iterations), it.w, it.h,
                            mine == k ? it.alive[g - s_prefix[k]] : kEmpty, stage[threadIdx.x / 32]);
            todo &= ~__ballot_sync(0xffffffffu, mine == k);
        }
    }
}

__global__ void advance_state_batch_kernel(const SiteBatchItem* __restrict__ items, uint32_t n_items,
                                           uint32_t vpt_passes, float beta1, float beta2) {
    pdl_wait();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_items) return;
    DevState* state = items[k].state;
    state->iter += 1u;
    state->vpt_pass += vpt_passes;
    set_bias_corrections(state, beta1, beta2);
}

static unsigned batch_grid(uint32_t grid_threads) { return std::max(1u, blocks_for(grid_threads, 256)); }

void launch_tau_first_batch(const SiteBatchItem* items, const uint32_t* site_prefix, uint32_t n_items, int field,
                            int iterations, uint32_t grid_threads, cudaStream_t st) {
    launch_pdl(tau_first_batch_kernel, dim3(batch_grid(grid_threads)), dim3(256), 0, st, items, site_prefix, n_items,
               field, iterations);
    note_launches(1);
}

void launch_tau_list_batch(const SiteBatchItem* items, const uint32_t* site_prefix, uint32_t n_items, bool a_to_b,
                           int iterations, uint32_t grid_threads, cudaStream_t st) {
    launch_pdl(tau_list_batch_kernel, dim3(batch_grid(grid_threads)), dim3(256), 0, st, items, site_prefix, n_items,
               a_to_b ? 1 : 0, iterations);
    note_launches(1);
}

void launch_adam_batch(const SiteBatchItem* items, const uint32_t* site_prefix, uint32_t n_items,
                       const AdamHyper& hp, int iterations, uint32_t grid_threads, cudaStream_t st) {
    launch_pdl(adam_batch_kernel, dim3(std::max(1u, blocks_for(grid_threads, kAdamThreads))), dim3(kAdamThreads), 0,
               st, items, site_prefix, n_items, hp, iterations);
    note_launches(1);
}

void launch_advance_state_batch(const SiteBatchItem* items, uint32_t n_items, uint32_t vpt_passes, float beta1,
                                float beta2, cudaStream_t st) {
    launch_pdl(advance_state_batch_kernel, dim3(blocks_for(n_items, 128)), dim3(128), 0, st, items, n_items,
               vpt_passes, beta1, beta2);
    note_launches(1);
}

}  // namespace sad

using namespace sad;

extern "C" sad_status_t sad_tau_diffuse(const uint32_t* cand0, const uint32_t* cand1,
                                        const float* sites, const float* grad_raw,
                                        const float* grad_in, float* grad_out, uint32_t site_count,
                                        float lambda, int width, int height, int cand_downscale,
                                        sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(image_size_ok(width, height), "sad_tau_diffuse: invalid cand size");
    SAD_REQUIRE(site_count == 0 || (cand0 && cand1 && sites && grad_raw && grad_in && grad_out),
                "sad_tau_diffuse: null buffer");
    SAD_REQUIRE(grad_in != grad_out, "sad_tau_diffuse: grad_in and grad_out must differ");
    launch_tau_diffuse_raw(cand0, cand1, reinterpret_cast<const Site*>(sites), grad_raw, grad_in,
                           grad_out, site_count, lambda, width, height, cand_downscale,
                           as_stream(stream));
    return check_launch("sad_tau_diffuse");
}

extern "C" sad_status_t sad_adam_update(float* sites, float* adam, const float* gpx,
                                        const float* gpy, const float* glt, const float* grad,
                                        const float* gr, const float* gg, const float* gb,
                                        const float* gdx, const float* gdy, const float* gla,
                                        float lr_pos, float lr_tau, float lr_radius,
                                        float lr_color, float lr_dir, float lr_aniso, float beta1,
                                        float beta2, float eps, uint32_t t, uint32_t site_count,
                                        int width, int height, sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(image_size_ok(width, height), "sad_adam_update: invalid image size");
    SAD_REQUIRE(site_count == 0 || (sites && adam && gpx && gpy && glt && grad && gr && gg && gb &&
                                    gdx && gdy && gla),
                "sad_adam_update: null buffer");
    SAD_REQUIRE((reinterpret_cast<uintptr_t>(adam) & 15u) == 0, "sad_adam_update: adam must be 16-byte aligned");
    AdamHyper hp{lr_pos, lr_tau, lr_radius, lr_color, lr_dir, lr_aniso, beta1, beta2, eps};
    const float* g[10] = {gpx, gpy, glt, grad, gr, gg, gb, gdx, gdy, gla};
    launch_adam_soa(reinterpret_cast<Site*>(sites), adam, g, hp, t, site_count, width, height,
                    as_stream(stream));
    return check_launch("sad_adam_update");
}

extern "C" sad_status_t sad_clear_gradients(float* g0, float* g1, float* g2, float* g3, float* g4,
                                            float* g5, float* g6, float* g7, float* g8, float* g9,
                                            uint32_t count, sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(count == 0 || (g0 && g1 && g2 && g3 && g4 && g5 && g6 && g7 && g8 && g9),
                "sad_clear_gradients: null buffer");
    if (count == 0) return SAD_OK;
    SoaGrads g{{g0, g1, g2, g3, g4, g5, g6, g7, g8, g9}};
    clear10_kernel<<<blocks_for(count, 256), 256, 0, as_stream(stream)>>>(g, count);
    note_launches(1);
    return check_launch("sad_clear_gradients");
}

extern "C" sad_status_t sad_clear_buffer(float* buffer, uint32_t count, sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(count == 0 || buffer, "sad_clear_buffer: null buffer");
    if (count == 0) return SAD_OK;
    return check_cuda(cudaMemsetAsync(buffer, 0, static_cast<size_t>(count) * sizeof(float), as_stream(stream)),
                      "sad_clear_buffer");
}

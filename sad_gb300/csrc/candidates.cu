// candidates.cu -- per-pixel candidate lists: f16 site packing, jump flooding (top-4) and
// the VPT propagation pass (top-8).
//
// Candidate distances are the reference's: tau_c * dmix2 with tau_c = max(exp(log_tau),
// 1e-4) (backends/cuda/src/jfa.cu:14-63, 150-174), evaluated on f16-rounded site values in
// the VPT pass.  The insertion rule is the reference's: a candidate already in the list
// is skipped, otherwise it takes the first slot whose distance is strictly larger.  Lists
// live in registers; insertion is a branch-free compare/select network.
#include "accum.cuh"
#include "common.cuh"
#include "host_common.h"
#include "kernels.h"

namespace sad {

// ---------------------------------------------------------------------------
// f16 packing (backends/cuda/src/candidate_pack.cu:3-28)
// ---------------------------------------------------------------------------
__global__ void pack_sites_kernel(const Site* __restrict__ sites, uint4* __restrict__ packed,
                                  uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2* q = reinterpret_cast<const float2*>(sites + i);
    float2 a = q[0], b = q[1], d = q[3], e = q[4];
    __half2 h0, h1, h2, h3;
    if (a.x < 0.0f) {
        __half neg = __float2half(-1.0f), z = __float2half(0.0f);
        h0 = __halves2half2(neg, neg);
        h1 = h2 = h3 = __halves2half2(z, z);
    } else {
        h0 = __halves2half2(__float2half(a.x), __float2half(a.y));
        h1 = __halves2half2(__float2half(b.x), __float2half(b.y));
        h2 = __halves2half2(__float2half(d.y), __float2half(e.x));
        h3 = __halves2half2(__float2half(e.y), __float2half(0.0f));
    }
    uint4 o;
    o.x = *reinterpret_cast<uint32_t*>(&h0);
    o.y = *reinterpret_cast<uint32_t*>(&h1);
    o.z = *reinterpret_cast<uint32_t*>(&h2);
    o.w = *reinterpret_cast<uint32_t*>(&h3);
    packed[i] = o;
}

void launch_pack_sites(const Site* sites, uint16_t* packed, uint32_t n, cudaStream_t st) {
    if (n == 0) return;
    pack_sites_kernel<<<blocks_for(n, 256), 256, 0, st>>>(sites, reinterpret_cast<uint4*>(packed), n);
    note_launches(1);
}

// Metric record of an f16 packed site: tau field = max(exp(log_tau), 1e-4).
__device__ __forceinline__ SiteGeom geom_from_packed(uint4 v) {
    __half2 h0 = *reinterpret_cast<__half2*>(&v.x);
    __half2 h1 = *reinterpret_cast<__half2*>(&v.y);
    __half2 h2 = *reinterpret_cast<__half2*>(&v.z);
    __half2 h3 = *reinterpret_cast<__half2*>(&v.w);
    float2 pos = __half22float2(h0), tr = __half22float2(h1), dir = __half22float2(h2),
           an = __half22float2(h3);
    SiteGeom g = make_geom(pos.x, pos.y, tr.x, tr.y, dir.x, dir.y, an.x);
    g.tau = fmaxf(g.tau, 1e-4f);
    return g;
}

// Trainer form: the same record built once per site per refresh (32-byte gathers in the
// pass instead of 16-byte gathers plus two expf and a division per visit).
__device__ __forceinline__ void pack_geom_one(const Site* __restrict__ sites, SiteGeom* __restrict__ out,
                                              uint32_t i);

__global__ void pack_geom_kernel(const Site* __restrict__ sites, SiteGeom* __restrict__ out,
                                 uint32_t n) {
    pdl_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    pack_geom_one(sites, out, i);
}

// The trainer's refresh: only the listed (active) sites; a pruned site's record is marked
// inactive by the prune itself.
__global__ void pack_geom_alive_kernel(const Site* __restrict__ sites, SiteGeom* __restrict__ out,
                                       const uint32_t* __restrict__ alive, const DevState* __restrict__ state) {
    pdl_wait();
    const uint32_t n_alive = state->n_alive;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n_alive; j += gridDim.x * blockDim.x)
        pack_geom_one(sites, out, alive[j]);
}

__device__ __forceinline__ void pack_geom_one(const Site* __restrict__ sites, SiteGeom* __restrict__ out,
                                              uint32_t i) {
    const float2* q = reinterpret_cast<const float2*>(sites + i);
    float2 a = q[0], b = q[1], d = q[3], e = q[4];
    uint4 v;
    if (a.x < 0.0f) {
        __half neg = __float2half(-1.0f), z = __float2half(0.0f);
        __half2 h0 = __halves2half2(neg, neg), hz = __halves2half2(z, z);
        v.x = *reinterpret_cast<uint32_t*>(&h0);
        v.y = v.z = v.w = *reinterpret_cast<uint32_t*>(&hz);
    } else {
        __half2 h0 = __halves2half2(__float2half(a.x), __float2half(a.y));
        __half2 h1 = __halves2half2(__float2half(b.x), __float2half(b.y));
        __half2 h2 = __halves2half2(__float2half(d.y), __float2half(e.x));
        __half2 h3 = __halves2half2(__float2half(e.y), __float2half(0.0f));
        v.x = *reinterpret_cast<uint32_t*>(&h0);
        v.y = *reinterpret_cast<uint32_t*>(&h1);
        v.z = *reinterpret_cast<uint32_t*>(&h2);
        v.w = *reinterpret_cast<uint32_t*>(&h3);
    }
    store_geom(out, i, geom_from_packed(v));
}

void launch_pack_geom(const Site* sites, SiteGeom* out, uint32_t n, cudaStream_t st) {
    if (n == 0) return;
    launch_pdl(pack_geom_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, st, sites, out, n);
    note_launches(1);
}

__global__ void __launch_bounds__(256) pack_geom_batch_kernel(const SiteBatchItem* __restrict__ items,
                                                              const uint32_t* __restrict__ prefix,
                                                              uint32_t n_items) {
    pdl_wait();
    __shared__ uint32_t s_prefix[kMaxBatchItems + 1];
    const uint32_t total = load_site_prefix(s_prefix, prefix, n_items);
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const uint32_t k = batch_item_of(s_prefix, n_items, g);
        const SiteBatchItem& it = items[k];
        pack_geom_one(it.sites, it.vgeom, it.alive[g - s_prefix[k]]);
    }
}

void launch_pack_geom_batch(const SiteBatchItem* items, const uint32_t* site_prefix, uint32_t n_items,
                            uint32_t grid_threads, cudaStream_t st) {
    launch_pdl(pack_geom_batch_kernel, dim3(std::max(1u, blocks_for(grid_threads, 256))), dim3(256), 0, st, items,
               site_prefix, n_items);
    note_launches(1);
}

void launch_pack_geom_alive(const Site* sites, SiteGeom* out, const uint32_t* alive, const DevState* state,
                            uint32_t max_alive, cudaStream_t st) {
    if (max_alive == 0) return;
    launch_pdl(pack_geom_alive_kernel, dim3(blocks_for(max_alive, 256)), dim3(256), 0, st, sites, out, alive,
               state);
    note_launches(1);
}

// The records of packed sites, once per site and call instead of once per visit.
__global__ void unpack_geom_kernel(const uint4* __restrict__ packed, SiteGeom* __restrict__ out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) store_geom(out, i, geom_from_packed(packed[i]));
}

static void launch_unpack_geom(const uint16_t* packed, SiteGeom* out, uint32_t n, cudaStream_t st) {
    if (n == 0) return;
    unpack_geom_kernel<<<blocks_for(n, 256), 256, 0, st>>>(reinterpret_cast<const uint4*>(packed), out, n);
    note_launches(1);
}

struct PackedHalfSites {
    const uint4* p;
    __device__ __forceinline__ SiteGeom load(uint32_t id) const { return geom_from_packed(__ldg(p + id)); }
};
struct PackedGeomSites {
    const SiteGeom* g;
    __device__ __forceinline__ SiteGeom load(uint32_t id) const { return load_geom(g, id); }
};

// ---------------------------------------------------------------------------
// sorted top-L lists
// ---------------------------------------------------------------------------
template <int L>
__device__ __forceinline__ void sorted_insert(uint32_t (&bi)[L], float (&bd)[L], uint32_t id,
                                              float d) {
    if (!(d < bd[L - 1])) return;  // not better than the last entry: no slot takes it
#pragma unroll
    for (int j = L - 1; j > 0; --j) {
        bool before_prev = d < bd[j - 1];
        bool before_this = d < bd[j];
        float nd = before_prev ? bd[j - 1] : (before_this ? d : bd[j]);
        uint32_t ni = before_prev ? bi[j - 1] : (before_this ? id : bi[j]);
        bd[j] = nd;
        bi[j] = ni;
    }
    if (d < bd[0]) {
        bd[0] = d;
        bi[0] = id;
    }
}

template <int L>
__device__ __forceinline__ bool in_list(const uint32_t (&bi)[L], uint32_t id) {
    bool hit = false;
#pragma unroll
    for (int j = 0; j < L; ++j) hit |= bi[j] == id;
    return hit;
}

// ---------------------------------------------------------------------------
// VPT pass
// ---------------------------------------------------------------------------
// The list a pass writes is the first eight, by distance and then by order of arrival, of
// the distinct active sites that arrive (insertClosest8Packed, backends/cuda/src/jfa.cu:
// 176-248): own list, four neighbours, radius probes, Hilbert probes, injected sites.  Most
// arrivals repeat an entry of the own list, so the pass works in three steps that keep that
// order:
//   1. the own list: eight distances at once, then adjacent exchanges until it is sorted
//      (none for a list that the last pass wrote and whose sites stayed);
//   2. of each neighbour's list, the ids that are not in the list yet go to the thread's
//      queue in shared memory (eight compares each, no load);
//   3. the queue is drained: distance, and insertion where it beats the last entry.
// An id that has been displaced, or turned down, can be queued again: its distance is not
// below the last entry's any more, so it is turned down again.
// Bound by issue and the L1 pipe (random gathers of the injected sites).  A late pass of a
// 1024x1024 render (8,192 sites) issues 49.7 M instead of 62.5 M warp instructions against
// inserting every arrival in turn, 74 instead of 84 us (ncu); twelve passes over 512x512
// with 16,384 sites from random lists 588 instead of 683 us.
constexpr int kVptThreads = 256;
constexpr int kVptQueue = 16;  // two neighbours' lists

struct VptQueue {
    uint32_t* base;  // this thread's column of the block's [kVptQueue][kVptThreads] words
    uint32_t* end;

    template <int L>
    __device__ __forceinline__ void offer(const uint32_t (&bi)[L], uint32_t id, uint32_t n) {
        if (id < n && !in_list<L>(bi, id)) {
            *end = id;
            end += kVptThreads;
        }
    }
    template <int L>
    __device__ __forceinline__ void offer4(const uint32_t (&bi)[L], uint4 c, uint32_t n) {
        offer<L>(bi, c.x, n);
        offer<L>(bi, c.y, n);
        offer<L>(bi, c.z, n);
        offer<L>(bi, c.w, n);
    }
};

// Distance of a site, +inf for an inactive one (never inserted).
template <class Src>
__device__ __forceinline__ float vpt_distance(const Src& src, uint32_t id, float ux, float uy, float inv_s2,
                                              float inv_scale) {
    SiteGeom g = src.load(id);
    return g.px < 0.0f ? INFINITY : g.tau * dmix2(g, ux, uy, inv_s2, inv_scale);
}

__device__ __forceinline__ void vpt_take(uint32_t (&bi)[8], float (&bd)[8], uint32_t id, float d) {
    if (d < bd[7] && !in_list<8>(bi, id)) sorted_insert<8>(bi, bd, id, d);
}

// Two sites at a time, so that their loads overlap (an odd last one pairs with itself).
template <class Src>
__device__ __forceinline__ void vpt_drain(VptQueue& q, uint32_t (&bi)[8], float (&bd)[8], float ux, float uy,
                                          const Src& src, float inv_s2, float inv_scale) {
#pragma unroll 1
    for (uint32_t* p = q.base; p < q.end; p += 2 * kVptThreads) {
        const uint32_t a = p[0];
        const uint32_t b = p + kVptThreads < q.end ? p[kVptThreads] : a;
        const float da = vpt_distance(src, a, ux, uy, inv_s2, inv_scale);
        const float db = vpt_distance(src, b, ux, uy, inv_s2, inv_scale);
        vpt_take(bi, bd, a, da);
        vpt_take(bi, bd, b, db);
    }
    q.end = q.base;
}

// The own list, sorted by distance (equal distances keep their order); repeated ids, ids
// past n and sites without a finite distance leave an empty entry at the end.
template <int L, class DistFn>
__device__ __forceinline__ void sorted_own_list(uint32_t (&bi)[L], float (&bd)[L], uint32_t n, DistFn dist) {
#pragma unroll
    for (int i = 0; i < L; ++i) {
        bool skip = bi[i] >= n;
#pragma unroll
        for (int j = 0; j < i; ++j) skip |= bi[j] == bi[i];
        bd[i] = skip ? INFINITY : dist(bi[i]);
    }
    bool again = false;
#pragma unroll
    for (int i = 0; i < L; ++i) {
        if (!(bd[i] < INFINITY)) {
            bd[i] = INFINITY;
            bi[i] = kEmpty;
        }
        if (i > 0) again |= bd[i - 1] > bd[i];
    }
#pragma unroll 1
    while (again) {
#pragma unroll
        for (int odd = 0; odd < 2; ++odd) {
#pragma unroll
            for (int i = odd; i + 1 < L; i += 2) {
                const bool swap = bd[i] > bd[i + 1];
                const float lo = swap ? bd[i + 1] : bd[i], hi = swap ? bd[i] : bd[i + 1];
                const uint32_t il = swap ? bi[i + 1] : bi[i], ih = swap ? bi[i] : bi[i + 1];
                bd[i] = lo;
                bd[i + 1] = hi;
                bi[i] = il;
                bi[i + 1] = ih;
            }
        }
        again = false;
#pragma unroll
        for (int i = 1; i < L; ++i) again |= bd[i - 1] > bd[i];
    }
}

// Jump schedule on the device (jumpStepForIndex/packJumpStep, sad_cuda.cu:1157-1183);
// pow2 and stages depend only on the field size and come from the host.
__device__ __forceinline__ uint32_t device_pack_jump(uint32_t idx, uint32_t pow2, uint32_t stages) {
    uint32_t jump = 1;
    if (pow2 > 1u) {
        uint32_t stage = idx >= stages ? stages - 1u : idx;
        jump = max(pow2 >> (stage + 1u), 1u);
    }
    jump = min(jump, 0xffffu);
    return (jump << 16) | (idx & 0xffffu);
}

// One VPT pass at candidate-field texel (x, y) (in range): writes the new list to
// prm.out0/out1.  backends/cuda/src/jfa.cu:271-386.
template <class Src>
__device__ __forceinline__ void vpt_pixel(const VptParams& prm, const Src& src, int x, int y, VptQueue q) {
    const int w = prm.width, h = prm.height;
    uint32_t step = prm.step, step_high = prm.step_high;
    if (prm.state) {
        uint32_t idx = prm.state->vpt_pass + prm.pass_offset;
        step = device_pack_jump(idx, prm.pow2, prm.stages);
        step_high = idx >> 16;
    }
    const uint32_t n = prm.site_count;
    uint32_t step_index = step & 0xffffu;
    uint32_t jump = step >> 16;
    if (jump == 0u) jump = 1u;
    uint32_t full_step = (step_high << 16) | step_index;
    float ux = fminf(static_cast<float>(x) * static_cast<float>(prm.cand_downscale),
                     static_cast<float>(prm.target_width - 1));
    float uy = fminf(static_cast<float>(y) * static_cast<float>(prm.cand_downscale),
                     static_cast<float>(prm.target_height - 1));
    const float inv_s2 = prm.inv_scale_sq;
    const float inv_scale = sqrtf(inv_s2);
    const uint4* in0 = reinterpret_cast<const uint4*>(prm.in0);
    const uint4* in1 = reinterpret_cast<const uint4*>(prm.in1);
    const int p = y * w + x;

    uint32_t bi[8];
    float bd[8];
    {
        const uint4 a = __ldg(in0 + p), b = __ldg(in1 + p);
        bi[0] = a.x; bi[1] = a.y; bi[2] = a.z; bi[3] = a.w;
        bi[4] = b.x; bi[5] = b.y; bi[6] = b.z; bi[7] = b.w;
    }
    if (prm.have_distances) {
        const float4 a = prm.distances[2 * p], b = prm.distances[2 * p + 1];
        bd[0] = a.x; bd[1] = a.y; bd[2] = a.z; bd[3] = a.w;
        bd[4] = b.x; bd[5] = b.y; bd[6] = b.z; bd[7] = b.w;
    } else {
        sorted_own_list<8>(bi, bd, n, [&](uint32_t id) { return vpt_distance(src, id, ux, uy, inv_s2, inv_scale); });
    }

    const int j = static_cast<int>(jump);
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {  // left and right, then up and down
        int qa, qb;
        if (k == 0) {
            qa = y * w + clampi(x - j, 0, w - 1);
            qb = y * w + clampi(x + j, 0, w - 1);
        } else {
            qa = clampi(y - j, 0, h - 1) * w + x;
            qb = clampi(y + j, 0, h - 1) * w + x;
        }
        const uint4 a0 = __ldg(in0 + qa), a1 = __ldg(in1 + qa), b0 = __ldg(in0 + qb), b1 = __ldg(in1 + qb);
        q.offer4<8>(bi, a0, n);
        q.offer4<8>(bi, a1, n);
        q.offer4<8>(bi, b0, n);
        q.offer4<8>(bi, b1, n);
        vpt_drain(q, bi, bd, ux, uy, src, inv_s2, inv_scale);
    }
    if (prm.radius_probes > 0u) {
        float rad = prm.radius_scale * (static_cast<float>(w) / 1024.0f);
        uint32_t st = (static_cast<uint32_t>(x) * 73856093u) ^ (static_cast<uint32_t>(y) * 19349663u) ^
                      ((step_index + jump) * 83492791u);
#pragma unroll 1
        for (uint32_t r = 0; r < prm.radius_probes; ++r) {
            st = xorshift32(st);
            float a = static_cast<float>(st) * (1.0f / 4294967296.0f) * 6.2831853f;
            int ddx = static_cast<int>(cosf(a) * rad);
            int ddy = static_cast<int>(sinf(a) * rad);
            int px = clampi(x + ddx, 0, w - 1), py = clampi(y + ddy, 0, h - 1);
            if (px == x && py == y) continue;
            const int qp = py * w + px;
            q.offer4<8>(bi, __ldg(in0 + qp), n);
            q.offer4<8>(bi, __ldg(in1 + qp), n);
            vpt_drain(q, bi, bd, ux, uy, src, inv_s2, inv_scale);
        }
    }
    if (prm.hilbert_probes > 0u && prm.hilbert_window > 0u) {
        uint32_t best = bi[0];
        if (best < n) {
            uint32_t pos = __ldg(prm.hilbert_pos + best);
            uint32_t span = prm.hilbert_window * 2u + 1u;
            uint32_t hs = (static_cast<uint32_t>(x) * 2654435761u) ^
                          (static_cast<uint32_t>(y) * 1597334677u) ^ (full_step * 374761393u);
#pragma unroll 1
            for (uint32_t i = 0; i < prm.hilbert_probes; ++i) {
                hs = xorshift32(hs + i);
                int o = static_cast<int>(hs % span) - static_cast<int>(prm.hilbert_window);
                int idx = clampi(static_cast<int>(pos) + o, 0, static_cast<int>(n - 1));
                const uint32_t id = __ldg(prm.hilbert_order + idx);
                if (id < n) vpt_take(bi, bd, id, vpt_distance(src, id, ux, uy, inv_s2, inv_scale));
            }
        }
    }
    uint32_t is = (static_cast<uint32_t>(x) * 1664525u) ^ (static_cast<uint32_t>(y) * 1013904223u) ^
                  (full_step * 374761393u);
#pragma unroll 1
    for (uint32_t i = 0; i < prm.inject_count; i += 2) {  // two at a time, as vpt_drain
        is = xorshift32(is + i);
        const uint32_t a = is % n;
        uint32_t b = a;
        if (i + 1 < prm.inject_count) {
            is = xorshift32(is + i + 1);
            b = is % n;
        }
        const float da = vpt_distance(src, a, ux, uy, inv_s2, inv_scale);
        const float db = vpt_distance(src, b, ux, uy, inv_s2, inv_scale);
        vpt_take(bi, bd, a, da);
        vpt_take(bi, bd, b, db);
    }
    reinterpret_cast<uint4*>(prm.out0)[p] = make_uint4(bi[0], bi[1], bi[2], bi[3]);
    reinterpret_cast<uint4*>(prm.out1)[p] = make_uint4(bi[4], bi[5], bi[6], bi[7]);
    if (prm.keep_distances) {
        prm.distances[2 * p] = make_float4(bd[0], bd[1], bd[2], bd[3]);
        prm.distances[2 * p + 1] = make_float4(bd[4], bd[5], bd[6], bd[7]);
    }
}

// Pixel of a thread in a 32x8-pixel block of eight warps: each warp takes an 8x4 patch, whose
// lanes share more of their sites than a 32x1 row's (fewer cache lines per gather, fewer
// lanes that differ at a branch).
__device__ __forceinline__ int2 patch_pixel(int block_x, int block_y) {
    const int lane = threadIdx.x, warp = threadIdx.y;
    return make_int2(block_x * 32 + (warp & 3) * 8 + (lane & 7), block_y * 8 + (warp >> 2) * 4 + (lane >> 3));
}

// This thread's column of the block's queue words.
__device__ __forceinline__ VptQueue thread_queue(uint32_t* words) {
    uint32_t* p = words + threadIdx.y * 32 + threadIdx.x;
    return VptQueue{p, p};
}

template <class Src>
__global__ void __launch_bounds__(kVptThreads, 5) vpt_kernel(VptParams prm, Src src) {
    __shared__ uint32_t s_queue[kVptQueue * kVptThreads];
    pdl_wait();
    const int2 at = patch_pixel(blockIdx.x, blockIdx.y);
    if (at.x >= prm.width || at.y >= prm.height) return;
    vpt_pixel(prm, src, at.x, at.y, thread_queue(s_queue));
}

// Batched form over the 32x8-pixel blocks of every image of a batch (the trainer's
// refresh pass on the f16-rounded geometry).
// The pass reads its parameters throughout each pixel's merges; one thread copies the
// block's image from the kernel parameters into shared memory (measured 3% faster than
// reading them from the constant bank, unlike the gradient kernel, whose shared-memory
// pipe is busy with the tile table's atomics).
__global__ void __launch_bounds__(kVptThreads, 5)
    vpt_batch_kernel(const __grid_constant__ BatchArgs<VptBatchItem> a) {
    __shared__ uint32_t s_queue[kVptQueue * kVptThreads];
    pdl_wait();
    __shared__ VptParams s_p;
    __shared__ const SiteGeom* s_g;
    __shared__ int s_local, s_bx;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        const uint32_t i = a.item_of(blockIdx.x);
        s_p = a.items[i].p;
        s_g = a.items[i].vgeom;
        s_bx = a.items[i].blocks_x;
        s_local = static_cast<int>(blockIdx.x - a.block_prefix[i]);
    }
    __syncthreads();
    const int2 at = patch_pixel(s_local % s_bx, s_local / s_bx);
    if (at.x >= s_p.width || at.y >= s_p.height) return;
    vpt_pixel(s_p, PackedGeomSites{s_g}, at.x, at.y, thread_queue(s_queue));
}

void launch_vpt_batch(const VptBatchItem* items, const uint32_t* block_prefix, uint32_t n_items, cudaStream_t st) {
    for_each_batch_launch(items, block_prefix, n_items, [&](const BatchArgs<VptBatchItem>& a, uint32_t blocks) {
        launch_pdl(vpt_batch_kernel, dim3(blocks), dim3(32, 8), 0, st, a);
        note_launches(1);
    });
}

static dim3 pixel_grid(int w, int h) { return dim3((w + 31) / 32, (h + 7) / 8); }

void launch_vpt_packed(const VptParams& prm, const uint16_t* packed, cudaStream_t st) {
    launch_pdl(vpt_kernel<PackedHalfSites>, pixel_grid(prm.width, prm.height), dim3(32, 8), 0, st,
        prm, PackedHalfSites{reinterpret_cast<const uint4*>(packed)});
    note_launches(1);
}

void launch_vpt_geom(const VptParams& prm, const SiteGeom* geom, cudaStream_t st) {
    launch_pdl(vpt_kernel<PackedGeomSites>, pixel_grid(prm.width, prm.height), dim3(32, 8), 0, st,
        prm, PackedGeomSites{geom});
    note_launches(1);
}

// ---------------------------------------------------------------------------
// JFA (backends/cuda/src/jfa.cu:66-144)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int seed_texel(float px, float py, int w, int h, int ds) {
    float inv = 1.0f / fmaxf(static_cast<float>(ds), 1.0f);
    int x = clampi(static_cast<int>(px * inv), 0, w - 1);
    int y = clampi(static_cast<int>(py * inv), 0, h - 1);
    return y * w + x;
}

// Two phases give a deterministic winner (the lowest id) where sites share a texel.
__global__ void jfa_seed_mark_kernel(uint32_t* __restrict__ cand0, const Site* __restrict__ sites,
                                     uint32_t n, int w, int h, int ds) {
    pdl_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float px = sites[i].px;
    if (px < 0.0f) return;
    cand0[4 * seed_texel(px, sites[i].py, w, h, ds)] = kEmpty;
}

__global__ void jfa_seed_min_kernel(uint32_t* __restrict__ cand0, const Site* __restrict__ sites,
                                    uint32_t n, int w, int h, int ds) {
    pdl_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float px = sites[i].px;
    if (px < 0.0f) return;
    atomicMin(&cand0[4 * seed_texel(px, sites[i].py, w, h, ds)], i);
}

void launch_jfa_seed(uint32_t* cand0, const Site* sites, uint32_t n, int w, int h, int ds,
                     cudaStream_t st) {
    if (n == 0) return;
    launch_pdl(jfa_seed_mark_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, st, cand0, sites, n, w, h, ds);
    launch_pdl(jfa_seed_min_kernel, dim3(blocks_for(n, 256)), dim3(256), 0, st, cand0, sites, n, w, h, ds);
    note_launches(2);
}

struct RawGeomSites {
    const Site* s;
    __device__ __forceinline__ SiteGeom load(uint32_t id) const {
        const float2* q = reinterpret_cast<const float2*>(s + id);
        float2 a = __ldg(q), b = __ldg(q + 1), d = __ldg(q + 3), e = __ldg(q + 4);
        return make_geom(a.x, a.y, b.x, b.y, d.y, e.x, e.y);
    }
};
struct FullGeomSites {
    const SiteGeom* g;
    __device__ __forceinline__ SiteGeom load(uint32_t id) const { return load_geom(g, id); }
};

// Distance of a site, +inf for an inactive one (never inserted).
template <class Src>
__device__ __forceinline__ float jfa_distance(const Src& src, uint32_t id, float ux, float uy, float inv_s2,
                                              float inv_scale) {
    SiteGeom g = src.load(id);
    return g.px < 0.0f ? INFINITY : fmaxf(g.tau, 1e-4f) * dmix2(g, ux, uy, inv_s2, inv_scale);
}

__device__ __forceinline__ bool in_quad(uint4 c, uint32_t id) {
    return c.x == id || c.y == id || c.z == id || c.w == id;
}

// Which texels a warp of a flood pass takes: 8x4 texels `stride` (1 << log2) apart in each
// direction.  The block's warps take neighbouring offsets, so together they still read whole
// lines: 8 offsets in x for a stride of 8 and more, 4 x 2 and 2 x 2 x 2 patches below that.
struct FloodTiling {
    int log2;
    __host__ __device__ int offsets_x() const { return log2 >= 3 ? 3 : log2; }          // log2 of the offsets per block
    __host__ __device__ int offsets_y() const { return log2 >= 3 ? 0 : log2 == 2 ? 1 : log2; }
    __host__ __device__ int patches() const { return 3 - offsets_x() - offsets_y(); }
    // texels covered by one block's column of patches, and the blocks that fill it
    __host__ __device__ int span_x() const { return 8 << (log2 + patches()); }
    __host__ __device__ int span_y() const { return 4 << log2; }
    __host__ __device__ int fill_x() const { return 1 << (log2 - offsets_x()); }
    __host__ __device__ int fill_y() const { return 1 << (log2 - offsets_y()); }

    __device__ __forceinline__ int2 texel(int bx, int by) const {
        const int lane = threadIdx.x, warp = threadIdx.y, ox = offsets_x(), oy = offsets_y();
        const int wx = warp & ((1 << ox) - 1), wy = (warp >> ox) & ((1 << oy) - 1), wp = warp >> (ox + oy);
        const int fx = log2 - ox, fy = log2 - oy;
        const int x = (bx >> fx) * span_x() + ((bx & ((1 << fx) - 1)) << ox) + wx + (wp * 8 + (lane & 7)) * (1 << log2);
        const int y = (by >> fy) * span_y() + ((by & ((1 << fy) - 1)) << oy) + wy + (lane >> 3) * (1 << log2);
        return make_int2(x, y);
    }
};

// One flood pass.  Until a pass of step s, sites have moved in steps of 2s and more: texels
// whose coordinates agree modulo 2s list sites of one set, and their neighbours in between
// list others.  Two things follow.
//   * Of the eight neighbours, left and right share a set, as do above and below and the
//     four corners.  An id that an earlier texel of its set has brought is skipped by four
//     compares per texel: it is in the list, or it was turned down or displaced and would be
//     again.  The others arrive in the reference's order through the queue.
//   * A warp takes texels 2s apart (FloodTiling), so its lanes gather the same few sites; of
//     32 adjacent texels each gathers its own.
// Bound by the L1 pipe (77-80% of its wavefronts) and issue.  A render from sites, against
// inserting all 36 arrivals of 32x1-texel warps in turn: 4096x4096 with 131,072 sites 34.9
// instead of 37.5 ms, 1024x1024 with 8,192 sites 2.03 instead of 2.07 ms (late passes 54 M
// instead of 63 M warp instructions).
template <class Src>
__global__ void __launch_bounds__(kVptThreads, 5) jfa_flood_kernel(const uint4* __restrict__ in0,
                                                                  uint4* __restrict__ out0, Src src,
                                                                  uint32_t n, uint32_t step_size, float inv_s2,
                                                                  int w, int h, int ds, int tw, int th,
                                                                  FloodTiling tiling) {
    __shared__ uint32_t s_queue[12 * kVptThreads];  // one row's lists
    pdl_wait();
    const int2 at = tiling.texel(blockIdx.x, blockIdx.z * gridDim.y + blockIdx.y);
    const int x = at.x, y = at.y;
    if (x >= w || y >= h) return;
    VptQueue q = thread_queue(s_queue);
    const float ux = fminf(static_cast<float>(x) * static_cast<float>(ds), static_cast<float>(tw - 1));
    const float uy = fminf(static_cast<float>(y) * static_cast<float>(ds), static_cast<float>(th - 1));
    const float inv_scale = sqrtf(inv_s2);
    const int step = static_cast<int>(step_size);
    uint32_t bi[4] = {kEmpty, kEmpty, kEmpty, kEmpty};
    float bd[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
    auto take = [&](uint32_t id, float d) {
        if (d < bd[3] && !in_list<4>(bi, id)) sorted_insert<4>(bi, bd, id, d);
    };
    auto drain = [&]() {
#pragma unroll 1
        for (uint32_t* p = q.base; p < q.end; p += 2 * kVptThreads) {
            const uint32_t e = p[0];
            const uint32_t f = p + kVptThreads < q.end ? p[kVptThreads] : e;
            const float de = jfa_distance(src, e, ux, uy, inv_s2, inv_scale);
            const float df = jfa_distance(src, f, ux, uy, inv_s2, inv_scale);
            take(e, de);
            take(f, df);
        }
        q.end = q.base;
    };
    // queues the ids of c for which seen() is false
    auto offer = [&](uint4 c, auto seen) {
        const uint32_t ids[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (ids[i] < n && !seen(ids[i])) {
                *q.end = ids[i];
                q.end += kVptThreads;
            }
        }
    };
    const auto none = [](uint32_t) { return false; };
    const int x0 = clampi(x - step, 0, w - 1), x1 = clampi(x + step, 0, w - 1);
    const int y0 = clampi(y - step, 0, h - 1) * w, yc = y * w, y1 = clampi(y + step, 0, h - 1) * w;
    const uint4 tl = __ldg(in0 + y0 + x0), tc = __ldg(in0 + y0 + x), tr = __ldg(in0 + y0 + x1);
    offer(tl, none);
    offer(tc, none);
    offer(tr, [&](uint32_t id) { return in_quad(tl, id); });
    drain();
    {
        const uint4 l = __ldg(in0 + yc + x0), c = __ldg(in0 + yc + x), r = __ldg(in0 + yc + x1);
        offer(l, none);
        offer(c, none);
        offer(r, [&](uint32_t id) { return in_quad(l, id); });
        drain();
    }
    {
        const uint4 bl = __ldg(in0 + y1 + x0), b = __ldg(in0 + y1 + x), br = __ldg(in0 + y1 + x1);
        offer(bl, [&](uint32_t id) { return in_quad(tl, id) || in_quad(tr, id); });
        offer(b, [&](uint32_t id) { return in_quad(tc, id); });
        offer(br, [&](uint32_t id) { return in_quad(tl, id) || in_quad(tr, id) || in_quad(bl, id); });
        drain();
    }
    out0[y * w + x] = make_uint4(bi[0], bi[1], bi[2], bi[3]);
}

// Stride of a pass: twice the step (the sites' sets), or the largest smaller power of two
// whose patches cover the field with at most a quarter of their texels outside.  While a set
// holds less than one site (n < 4 step^2) lists are mostly empty and reading them is the work:
// adjacent texels then (1024x1024, 8,192 sites: 21, 25 and 34 us for the steps 512, 256 and
// 128, against 35, 43 and 50 us strided; from step 32 on 77-87 us strided, 98-139 us adjacent).
static FloodTiling flood_tiling(uint32_t step, uint32_t n, int w, int h) {
    FloodTiling t{0};
    if (static_cast<double>(n) < 4.0 * step * step) return t;
    while (t.log2 < 14 && (2u << t.log2) <= 2u * step) ++t.log2;
    auto padded = [](int size, int span) { return static_cast<double>((size + span - 1) / span) * span; };
    while (t.log2 > 0 && padded(w, t.span_x()) * padded(h, t.span_y()) > 1.25 * w * h) --t.log2;
    return t;
}

template <class Src>
static void launch_jfa_flood(const uint32_t* in0, uint32_t* out0, Src src, uint32_t n, uint32_t step,
                             float inv_s2, int w, int h, int ds, int tw, int th, cudaStream_t st) {
    FloodTiling t = flood_tiling(step, n, w, h);
    // a block takes four rows at stride 1: past the limit of the grid's y the rows of blocks are
    // halved into z, so that a field may have 524,280 rows, as with eight a block
    const auto rows = [&] { return (h + t.span_y() - 1) / t.span_y() * t.fill_y(); };
    while (t.log2 > 0 && rows() > 2 * kMaxGridRows) --t.log2;
    const int folds = rows() > kMaxGridRows ? 2 : 1;
    const dim3 grid((w + t.span_x() - 1) / t.span_x() * t.fill_x(), (rows() + folds - 1) / folds, folds);
    launch_pdl(jfa_flood_kernel<Src>, grid, dim3(32, 8), 0, st, reinterpret_cast<const uint4*>(in0),
               reinterpret_cast<uint4*>(out0), src, n, step, inv_s2, w, h, ds, tw, th, t);
    note_launches(1);
}

void launch_jfa_flood_raw(const uint32_t* in0, uint32_t* out0, const Site* sites, uint32_t n,
                          uint32_t step, float inv_s2, int w, int h, int ds, int tw, int th,
                          cudaStream_t st) {
    launch_jfa_flood(in0, out0, RawGeomSites{sites}, n, step, inv_s2, w, h, ds, tw, th, st);
}

void launch_jfa_flood_geom(const uint32_t* in0, uint32_t* out0, const SiteGeom* geom, uint32_t n,
                           uint32_t step, float inv_s2, int w, int h, int ds, int tw, int th,
                           cudaStream_t st) {
    launch_jfa_flood(in0, out0, FullGeomSites{geom}, n, step, inv_s2, w, h, ds, tw, th, st);
}

uint32_t host_jump_step_for_index(uint32_t idx, int w, int h) {
    uint32_t maxd = static_cast<uint32_t>(w > h ? w : h);
    uint32_t pow2 = 1;
    while (pow2 < maxd) pow2 <<= 1;
    if (pow2 <= 1) return 1;
    uint32_t stages = 0, t = pow2;
    while (t > 1) {
        t >>= 1;
        ++stages;
    }
    uint32_t stage = idx >= stages ? stages - 1 : idx;
    uint32_t s = pow2 >> (stage + 1);
    return s > 1u ? s : 1u;
}

void jump_schedule_constants(int w, int h, uint32_t* pow2_out, uint32_t* stages_out) {
    uint32_t maxd = static_cast<uint32_t>(w > h ? w : h);
    uint32_t pow2 = 1;
    while (pow2 < maxd) pow2 <<= 1;
    uint32_t stages = 0, t = pow2;
    while (t > 1) {
        t >>= 1;
        ++stages;
    }
    *pow2_out = pow2;
    *stages_out = stages;
}

}  // namespace sad

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace sad;

extern "C" uint32_t sad_jump_step_for_index(uint32_t step_index, int width, int height) {
    return host_jump_step_for_index(step_index, width, height);
}

extern "C" uint32_t sad_pack_jump_step(uint32_t step_index, int width, int height) {
    uint32_t j = host_jump_step_for_index(step_index, width, height);
    if (j > 0xffffu) j = 0xffffu;
    return (j << 16) | (step_index & 0xffffu);
}

extern "C" sad_status_t sad_pack_candidate_sites(const float* sites, uint16_t* packed,
                                                 uint32_t site_count, sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(site_count == 0 || (sites && packed), "sad_pack_candidate_sites: null buffer");
    launch_pack_sites(reinterpret_cast<const Site*>(sites), packed, site_count, as_stream(stream));
    return check_launch("sad_pack_candidate_sites");
}

extern "C" sad_status_t sad_jfa_seed(uint32_t* cand0, const float* sites, uint32_t site_count,
                                     int width, int height, int cand_downscale,
                                     sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(image_size_ok(width, height), "sad_jfa_seed: invalid cand size");
    SAD_REQUIRE(cand0 && (sites || site_count == 0), "sad_jfa_seed: null buffer");
    launch_jfa_seed(cand0, reinterpret_cast<const Site*>(sites), site_count, width, height,
                    cand_downscale, as_stream(stream));
    return check_launch("sad_jfa_seed");
}

extern "C" sad_status_t sad_jfa_flood(const uint32_t* in_cand0, uint32_t* out_cand0,
                                      const float* sites, uint32_t site_count, uint32_t step_size,
                                      float inv_scale_sq, int width, int height,
                                      int cand_downscale, int target_width, int target_height,
                                      sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(image_size_ok(width, height), "sad_jfa_flood: invalid cand size");
    SAD_REQUIRE(target_width > 0 && target_height > 0, "sad_jfa_flood: invalid target size");
    SAD_REQUIRE(in_cand0 && out_cand0 && (sites || site_count == 0), "sad_jfa_flood: null buffer");
    SAD_REQUIRE(in_cand0 != out_cand0, "sad_jfa_flood: in and out must differ");
    launch_jfa_flood_raw(in_cand0, out_cand0, reinterpret_cast<const Site*>(sites), site_count,
                         step_size, inv_scale_sq, width, height, cand_downscale, target_width,
                         target_height, as_stream(stream));
    return check_launch("sad_jfa_flood");
}

// sites: raw sites (nullptr: packed_sites); records: scratch for a record per site (nullptr:
// the pass decodes packed_sites at every visit).
static sad_status_t update_candidates(
    const uint32_t* in_cand0, const uint32_t* in_cand1, uint32_t* out_cand0, uint32_t* out_cand1,
    const uint16_t* packed_sites, const float* sites, uint32_t site_count, uint32_t step, float inv_scale_sq,
    uint32_t step_high, float radius_scale, uint32_t radius_probes, uint32_t inject_count,
    const uint32_t* hilbert_order, const uint32_t* hilbert_pos, uint32_t hilbert_probes,
    uint32_t hilbert_window, int cand_downscale, int target_width, int target_height, int width,
    int height, SiteGeom* records, cudaStream_t stream) {
    SAD_REQUIRE(image_size_ok(width, height), "sad_update_candidates: invalid cand size");
    SAD_REQUIRE(target_width > 0 && target_height > 0, "sad_update_candidates: invalid target size");
    SAD_REQUIRE(in_cand0 && in_cand1 && out_cand0 && out_cand1, "sad_update_candidates: null field");
    SAD_REQUIRE(in_cand0 != out_cand0 && in_cand1 != out_cand1,
                "sad_update_candidates: in and out fields must differ");
    SAD_REQUIRE(site_count == 0 || packed_sites || sites, "sad_update_candidates: null packed sites");
    bool use_h = hilbert_probes > 0 && hilbert_window > 0;
    SAD_REQUIRE(!use_h || (hilbert_order && hilbert_pos),
                "sad_update_candidates: hilbert probes need hilbert_order and hilbert_pos");
    VptParams prm{};
    prm.in0 = in_cand0;
    prm.in1 = in_cand1;
    prm.out0 = out_cand0;
    prm.out1 = out_cand1;
    prm.site_count = site_count;
    prm.step = step;
    prm.step_high = step_high;
    prm.inv_scale_sq = inv_scale_sq;
    prm.radius_scale = radius_scale;
    prm.radius_probes = radius_probes;
    prm.inject_count = site_count == 0 ? 0u : inject_count;
    prm.hilbert_order = hilbert_order;
    prm.hilbert_pos = hilbert_pos;
    prm.hilbert_probes = use_h ? hilbert_probes : 0u;
    prm.hilbert_window = use_h ? hilbert_window : 0u;
    prm.cand_downscale = cand_downscale;
    prm.target_width = target_width;
    prm.target_height = target_height;
    prm.width = width;
    prm.height = height;
    prm.state = nullptr;
    if (!records) {
        launch_vpt_packed(prm, packed_sites, stream);
    } else {
        if (sites)
            launch_pack_geom(reinterpret_cast<const Site*>(sites), records, site_count, stream);
        else
            launch_unpack_geom(packed_sites, records, site_count, stream);
        launch_vpt_geom(prm, records, stream);
    }
    return check_launch("sad_update_candidates");
}

extern "C" sad_status_t sad_update_candidates(
    const uint32_t* in_cand0, const uint32_t* in_cand1, uint32_t* out_cand0, uint32_t* out_cand1,
    const uint16_t* packed_sites, uint32_t site_count, uint32_t step, float inv_scale_sq,
    uint32_t step_high, float radius_scale, uint32_t radius_probes, uint32_t inject_count,
    const uint32_t* hilbert_order, const uint32_t* hilbert_pos, uint32_t hilbert_probes,
    uint32_t hilbert_window, int cand_downscale, int target_width, int target_height, int width,
    int height, sad_stream_t stream) {
    clear_error();
    return update_candidates(in_cand0, in_cand1, out_cand0, out_cand1, packed_sites, nullptr, site_count, step,
                             inv_scale_sq, step_high, radius_scale, radius_probes, inject_count, hilbert_order,
                             hilbert_pos, hilbert_probes, hilbert_window, cand_downscale, target_width,
                             target_height, width, height, nullptr, as_stream(stream));
}

extern "C" size_t sad_update_candidates_scratch_bytes(uint32_t site_count) {
    return static_cast<size_t>(site_count) * sizeof(SiteGeom) + alignof(SiteGeom);
}

extern "C" sad_status_t sad_update_candidates_in(
    const uint32_t* in_cand0, const uint32_t* in_cand1, uint32_t* out_cand0, uint32_t* out_cand1,
    const uint16_t* packed_sites, const float* sites, uint32_t site_count, uint32_t step, float inv_scale_sq,
    uint32_t step_high, float radius_scale, uint32_t radius_probes, uint32_t inject_count,
    const uint32_t* hilbert_order, const uint32_t* hilbert_pos, uint32_t hilbert_probes,
    uint32_t hilbert_window, int cand_downscale, int target_width, int target_height, int width,
    int height, void* scratch, size_t scratch_bytes, sad_stream_t stream) {
    clear_error();
    SAD_REQUIRE(scratch && scratch_bytes >= sad_update_candidates_scratch_bytes(site_count),
                "sad_update_candidates_in: scratch too small");
    const uintptr_t base = (reinterpret_cast<uintptr_t>(scratch) + alignof(SiteGeom) - 1) & ~(alignof(SiteGeom) - 1);
    return update_candidates(in_cand0, in_cand1, out_cand0, out_cand1, packed_sites, sites, site_count, step,
                             inv_scale_sq, step_high, radius_scale, radius_probes, inject_count, hilbert_order,
                             hilbert_pos, hilbert_probes, hilbert_window, cand_downscale, target_width,
                             target_height, width, height, reinterpret_cast<SiteGeom*>(base), as_stream(stream));
}

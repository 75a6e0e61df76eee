// warp_sums.cuh -- per-site gradient sums of a warp's pixels, for the kernels that add into
// float arrays (the autograd adjoint and the tiled gradients of the API).
//
// Shared memory has no native float add: each one is a compare-and-swap loop, and lanes that
// list the same site queue up in it.  Here each group of eight lanes (a 4x2 patch of pixels,
// whose 64 candidates name some 10-20 distinct sites) takes one site after the other, the
// smallest id left first: the lanes that list it compute their terms, a folding butterfly
// sums them over the group and leaves each lane two of the sums at most, which go to global
// memory by one reduction per value.  No add in shared memory.
// What is the same for every pixel of a site (softness, scales) is multiplied in after the
// sum.  Groups of 8 balance the site loop's length, which falls with the group (fewer
// distinct sites, fewer idle lanes), against the global reductions, which rise: a 1999x1503
// render and its adjoint took 372 us (378 now), with groups of 4 and 16 lanes 481 and 468 us.
// A lane sorts its list by id first (19 exchanges), so that the loop compares and shifts its
// head instead of scanning eight ids for the minimum and for each match (some 20 of 150
// instructions a round): 372 instead of 394 us there from site records; a step at 1237x941 with
// SSIM and removal deltas 325 instead of 328 us.
// Lists with little in common (a random initial field) would make that loop long: a block with
// such a group (kMostMarks) takes a key table in shared memory instead, whose float adds rarely
// meet then (added straight to global memory, the terms' arbitrary order would show in more of
// the sums' last bits).  With few sites on many pixels all sums go that way (TableRule).
#pragma once

#include "accum.cuh"
#include "common.cuh"
#include "sources.cuh"

namespace sad {

constexpr int kSumGroup = 8;
constexpr int kSumSlots = 512;  // keys of the block's table

// Whether all sums go through the table: with few sites on many pixels the groups' reductions
// queue up at the same addresses in L2 (1999x1503 with 64 sites: the adjoint 2775 us, 759 by
// table; the gradients with SSIM and removal deltas 3978 and 893 us), and a table holds every
// site.  The line lies where the two meet on nearest-site fields: at one site per `per_site`
// pixels on small images and at `most` sites on large ones.  Adjoint by groups and by table: at
// 256x256 with 64 sites 75 and 45 us, with 100 sites 48 and 46; at 1024x1024 with 300 sites 362 and
// 317, with 400 sites 271 and 323.  Gradients: at 256x256 with 100 sites 79 and 53 us, with 256
// sites 46 and 55; at 1024x1024 with 300 sites 441 and 381, with 512 sites 374 and 392.
struct TableRule {
    int per_site;
    uint32_t most;
};
constexpr TableRule kAdjointTable = {1000, 300}, kGradientTable = {320, 400};
inline bool sums_by_table(const TableRule& rule, uint32_t n, int w, int h) {
    return n <= rule.most && static_cast<double>(w) * h >= static_cast<double>(rule.per_site) * n;
}

// Pixel of a lane in its warp's 8x4 patch, with every eight lanes a 4x2 patch.
__device__ __forceinline__ int2 sum_patch_pixel(int lane) {
    return make_int2((lane & 3) | ((lane >> 1) & 4), ((lane >> 2) & 1) | ((lane >> 3) & 2));
}

// Values left in a lane after folding N values over a group of G lanes.
template <int N, int G>
struct FoldedCount {
    static constexpr int value = FoldedCount<(N + 1) / 2, G / 2>::value;
};
template <int N>
struct FoldedCount<N, 1> {
    static constexpr int value = N;
};

// One half of the lanes keeps the first half of the values, the other half the rest, each
// summed over two lanes; then the same again within each half of the group.
template <int N, int G>
__device__ __forceinline__ void fold_values(const float (&v)[N], float (&r)[FoldedCount<N, G>::value], uint32_t lane) {
    if constexpr (G == 1) {
#pragma unroll
        for (int k = 0; k < N; ++k) r[k] = v[k];
    } else {
        constexpr int H = (N + 1) / 2;
        const bool upper = (lane & (G / 2)) != 0;
        float t[H];
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const float a = v[k], b = k + H < N ? v[k + H < N ? k + H : 0] : 0.0f;
            t[k] = (upper ? b : a) + __shfl_xor_sync(0xffffffffu, upper ? a : b, G / 2);
        }
        fold_values<H, G / 2>(t, r, lane);
    }
}

// The values that fold_values leaves in a lane are numbers first .. first + count - 1.
template <int N, int G>
__device__ __forceinline__ void folded_range(uint32_t lane, int& first, int& count) {
    int lo = 0, hi = N, size = N;
#pragma unroll
    for (int g = G; g > 1; g /= 2) {
        const int half = (size + 1) / 2;
        if (lane & (g / 2)) lo += half;
        else hi = min(hi, lo + half);
        size = half;
    }
    first = lo;
    count = max(0, min(hi - lo, size));
}

// Whether a zero weight's terms at this pixel are zeros (an infinity or NaN makes them NaN).
__device__ __forceinline__ bool zero_weight_adds_zeros(float3 dLdp, float3 pred) {
    return 0.0f * dLdp.x + 0.0f * dLdp.y + 0.0f * dLdp.z + 0.0f * pred.x + 0.0f * pred.y + 0.0f * pred.z == 0.0f;
}

// What one (pixel, site) adds to the site's sums, in the order of its parameters (position,
// log_tau, radius, colour, direction, log_aniso): candidate_grads without the factors that
// sum_scale() holds.
__device__ __forceinline__ void candidate_terms(const SiteGeom& g, float3 col, float ux, float uy, float inv_s2,
                                                float inv_scale, float w, float3 dLdp, float3 pred, float* v) {
    v[4] = w * dLdp.x;
    v[5] = w * dLdp.y;
    v[6] = w * dLdp.z;
    const float dlogit = v[4] * (col.x - pred.x) + v[5] * (col.y - pred.y) + v[6] * (col.z - pred.z);
    const float dx = ux - g.px, dy = uy - g.py;
    const float proj = g.dx * dx + g.dy * dy;
    const float proj2 = proj * proj;
    const float along = g.l1 * proj2, across = g.l2 * fmaxf(dx * dx + dy * dy - proj2, 0.0f);
    const float d2s = fmaxf((along + across) * inv_s2, 1e-8f);
    const float isq = rsqrtf(d2s);
    const float q = dlogit * isq;
    const float turn = (g.l1 - g.l2) * proj;
    v[0] = q * (g.l2 * dx + turn * g.dx);
    v[1] = q * (g.l2 * dy + turn * g.dy);
    v[2] = dlogit * (d2s * isq - g.radius * inv_scale);
    v[3] = dlogit;
    v[7] = q * turn * dx;
    v[8] = q * turn * dy;
    v[9] = q * (along - across);
}

// The constant factor of value k; times the site's tau where by_tau.
__device__ __forceinline__ float sum_scale(int k, float inv_s2, float inv_scale, bool& by_tau) {
    by_tau = k < 4 || (k >= 7 && k <= 9);
    if (k < 2) return inv_s2;
    if (k == 2) return -1.0f;
    if (k == 3) return inv_scale;
    if (k == 7 || k == 8) return -inv_s2;
    if (k == 9) return -0.5f * inv_s2;
    return 1.0f;
}

// Ascending ids, with what goes with them (Batcher's odd-even merge sort).
template <bool kRemoval>
__device__ __forceinline__ void sort_candidates(uint32_t (&ids)[kCand], float (&wts)[kCand], float (&rem)[kCand]) {
    const int net[19][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3}, {4, 6}, {5, 7}, {1, 2}, {5, 6},
                            {0, 4}, {1, 5}, {2, 6}, {3, 7}, {2, 4}, {3, 5}, {1, 2}, {3, 4}, {5, 6}};
    auto exchange = [](auto& a, auto& b, bool swap) {
        const auto lo = swap ? b : a, hi = swap ? a : b;
        a = lo;
        b = hi;
    };
#pragma unroll
    for (int e = 0; e < 19; ++e) {
        const int i = net[e][0], j = net[e][1];
        const bool swap = ids[i] > ids[j];
        exchange(ids[i], ids[j], swap);
        exchange(wts[i], wts[j], swap);
        if constexpr (kRemoval) exchange(rem[i], rem[j], swap);
    }
}

// How many of 64 hash values the ids of the lane's group take: 64 (1 - e^(-d/64)) for d distinct
// ids, give or take two.  Some 27 sites, or rounds of the loop, are its limit, which a field of
// one site a pixel still keeps: the adjoint at 256x256 with 65,536 sites takes 25 us with a
// limit of 22 marks, 46 with 19; at 512x512 with 262,144 sites 52 and 72 us; with a limit of
// 25 both the same.
constexpr int kMostMarks = 22;
__device__ __forceinline__ int distinct_marks(const uint32_t (&ids)[kCand]) {
    uint32_t lo = 0u, hi = 0u;
#pragma unroll
    for (int i = 0; i < kCand; ++i) {
        const uint32_t h = (ids[i] * 2654435761u) >> 26, bit = ids[i] == kEmpty ? 0u : 1u << (h & 31u);
        lo |= h & 32u ? 0u : bit;
        hi |= h & 32u ? bit : 0u;
    }
#pragma unroll
    for (int m = kSumGroup / 2; m > 0; m /= 2) {
        lo |= __shfl_xor_sync(0xffffffffu, lo, m);
        hi |= __shfl_xor_sync(0xffffffffu, hi, m);
    }
    return __popc(lo) + __popc(hi);
}

// Whether a warp of the block has left its pixels to the table: the others then leave the site
// loop, where they would keep it waiting.  begin_sums() before the first loads (a barrier later,
// where the warps have drifted apart, cost the adjoint at 1999x1503 4%).
__device__ __forceinline__ volatile int* block_takes_table() {
    __shared__ int s_takes_table;
    return &s_takes_table;
}
__device__ __forceinline__ void begin_sums(int tid) {
    if (tid == 0) *block_takes_table() = 0;
    __syncthreads();
}

// A pixel's candidates, for add_by_table.
struct PixelCandidates {
    uint32_t ids[kCand];
    float wts[kCand], rem[kCand];
    float ux, uy, inv_s2, inv_scale;
    float3 dLdp, pred;
};

// Adds a block's candidates through its key table (all 256 threads call it; ids: kEmpty where a
// slot carries none).  kArrays: add() goes to an array per value, where neighbouring lanes take
// neighbouring sites at the end, instead of neighbouring values of a site's row.
template <bool kRemoval, bool kArrays, class Load, class Add>
__device__ __forceinline__ void sum_by_table(uint32_t (&ids)[kCand], float (&wts)[kCand], float (&rem)[kCand],
                                             float ux, float uy, float inv_s2, float inv_scale, float3 dLdp,
                                             float3 pred, Load load, Add add) {
    constexpr int NV = kRemoval ? 11 : 10;
    __shared__ TileTable<NV, kSumSlots, AccFloat> table;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    table.init(tid, 256);
    __syncthreads();
    int slots[kCand];
#pragma unroll
    for (int i = 0; i < kCand; ++i) slots[i] = register_key(table, ids[i]);
    const uint32_t turn = lane_rotation();  // lanes with like lists visit different sites at a step
    rotate8(ids, turn);
    rotate8(wts, turn);
    rotate8(slots, turn);
    if constexpr (kRemoval) rotate8(rem, turn);
#pragma unroll 1
    for (int j = 0; j < kCand; ++j) {
        if (ids[0] != kEmpty) {
            SiteGeom g;
            float3 col;
            load(ids[0], g, col);
            float o[10], v[NV];
            candidate_grads(g, col, ux, uy, inv_s2, inv_scale, wts[0], dLdp, pred, false, o);
#pragma unroll
            for (int k = 0; k < 10; ++k) v[k] = o[k];
            if constexpr (kRemoval) v[10] = rem[0];
            if (slots[0] >= 0) {
                table.add(slots[0], v);
            } else {
#pragma unroll
                for (int k = 0; k < NV; ++k) add(ids[0], k, v[k]);
            }
        }
        shift8(ids);
        shift8(wts);
        shift8(slots);
        if constexpr (kRemoval) shift8(rem);
    }
    __syncthreads();
    const int used = table.size();
    if constexpr (kArrays) {
        for (int d = tid; d < used; d += 256) {
#pragma unroll
            for (int k = 0; k < NV; ++k) add(table.key_at(d), k, table.value(k, d));
        }
    } else {
        for (int q = tid; q < used * NV; q += 256) {
            const int d = q / NV, k = q - d * NV;
            add(table.key_at(d), k, table.value(k, d));
        }
    }
}

// The same as a call of its own, and with arguments of its own: inlined beside the site loop, its
// registers cost the loop 6% (1999x1503: 419 instead of 395 us).
template <bool kRemoval, bool kArrays, class Load, class Add>
__device__ __noinline__ void add_by_table(const PixelCandidates& from, Load load, Add add) {
    uint32_t ids[kCand];
    float wts[kCand], rem[kCand];
#pragma unroll
    for (int i = 0; i < kCand; ++i) {
        ids[i] = from.ids[i];
        wts[i] = from.wts[i];
        if constexpr (kRemoval) rem[i] = from.rem[i];
    }
    sum_by_table<kRemoval, kArrays>(ids, wts, rem, from.ux, from.uy, from.inv_s2, from.inv_scale, from.dLdp, from.pred,
                                    load, add);
}

// Adds the gradients of a block's pixels (all 256 threads call it; ids: kEmpty where a slot
// carries none).  load(id, geom, colour) reads a site; add(id, k, value) adds to value k of a
// site: its ten parameters and, with kRemoval, rem[] as value 10; by_table(from) calls
// add_by_table.
template <bool kRemoval, class Load, class Add, class Table>
__device__ __forceinline__ void add_site_gradients(uint32_t (&ids)[kCand], float (&wts)[kCand],
                                                   float (&rem)[kCand], float ux, float uy, float inv_s2,
                                                   float inv_scale, float3 dLdp, float3 pred, Load load, Add add,
                                                   Table by_table) {
    constexpr int NV = kRemoval ? 11 : 10, G = kSumGroup, R = FoldedCount<NV, G>::value;
    constexpr uint32_t full = 0xffffffffu;
    const uint32_t lane = lane_id();
    int first, count;
    folded_range<NV, G>(lane, first, count);
    float scale[R];
    bool by_tau[R];
#pragma unroll
    for (int k = 0; k < R; ++k) scale[k] = sum_scale(first + k, inv_s2, inv_scale, by_tau[k]);
    bool left = __any_sync(full, distinct_marks(ids) > kMostMarks);
    if (left) *block_takes_table() = 1;  // no loop in this warp, and soon none in the others
    else sort_candidates<kRemoval>(ids, wts, rem);
#pragma unroll 1
    while (!left) {
        const int stop = *block_takes_table();
        uint32_t id = ids[0];
#pragma unroll
        for (int m = G / 2; m > 0; m /= 2) id = min(id, __shfl_xor_sync(full, id, m));
        if (!__any_sync(full, id != kEmpty && stop == 0)) break;
        const bool mine = ids[0] == id && id != kEmpty;  // a repeated id comes again
        const float w = wts[0], r = kRemoval ? rem[0] : 0.0f;
        if (mine) {
            shift8(ids);
            shift8(wts);
            if constexpr (kRemoval) shift8(rem);
            ids[kCand - 1] = kEmpty;
        }
        float v[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] = 0.0f;
        float tau = 1.0f;
        if (id != kEmpty) {
            SiteGeom g;
            float3 col;
            load(id, g, col);
            tau = g.tau;
            if (mine) {
                candidate_terms(g, col, ux, uy, inv_s2, inv_scale, w, dLdp, pred, v);
                if constexpr (kRemoval) v[10] = r;
            }
        }
        float s[R];
        fold_values<NV, G>(v, s, lane);
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (k < count && id != kEmpty) add(id, first + k, s[k] * (scale[k] * (by_tau[k] ? tau : 1.0f)));
    }
    if (!__syncthreads_or(left || ids[0] != kEmpty)) return;
    PixelCandidates rest;
#pragma unroll
    for (int i = 0; i < kCand; ++i) {
        rest.ids[i] = ids[i];
        rest.wts[i] = wts[i];
        if constexpr (kRemoval) rest.rem[i] = rem[i];
    }
    rest.ux = ux;
    rest.uy = uy;
    rest.inv_s2 = inv_s2;
    rest.inv_scale = inv_scale;
    rest.dLdp = dLdp;
    rest.pred = pred;
    by_table(rest);
}

}  // namespace sad

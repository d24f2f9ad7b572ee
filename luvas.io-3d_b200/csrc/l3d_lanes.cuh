/*
 * The red/black propagate step with eight lanes per pixel, shared by the plain and the batched
 * forms' kernels, and the neighbour pattern both step kernels walk.
 *
 * A pixel's step (patchmatch.wgsl.ts:349-423) tries fourteen planes one after the other, each a
 * window in every source.  With a thread per pixel a small image leaves most of the chip idle while
 * every thread walks that chain (160x120: 75 blocks of 128 threads on 148 SMs).  But only two of the
 * fourteen steps depend on each other: the planes of the eight regions are given, and so are the six
 * refinements once the best of the eight is known.  So eight lanes take one candidate each, agree on
 * the winner, and six of them take the refinements: the chain is two planes long and there are
 * eight times the threads.  The window is prepared once by the eight lanes together.  What it
 * costs is a quarter of the lanes in the second round and the random numbers drawn eight times, so
 * launches that fill the chip anyway keep the thread per pixel (see the launchers' thresholds).
 */
#ifndef L3D_LANES_CUH
#define L3D_LANES_CUH

#include <stdint.h>
#include <cuda_runtime.h>

#include "l3d_fmath.h"

/* Offset i of a region: the near regions' seven pixels, turned into direction dir (0..3). */
__device__ __forceinline__ void l3d_near_offset(int i, int* ox, int* oy) {
    int m = (i + 1) / 2;
    *ox = (i & 1) ? -m : m;
    *oy = -(m + 1);
}
__device__ __forceinline__ void l3d_orient(int ox, int oy, int dir, int* rx, int* ry) {
    switch (dir) {
        case 1: *rx = ox; *ry = -oy; break;
        case 2: *rx = oy; *ry = ox; break;
        case 3: *rx = -oy; *ry = ox; break;
        default: *rx = ox; *ry = oy; break;
    }
}

/* The cheapest pixel of a region (0..3 near, 4..7 far along a line) around (x, y), -1 when none lies in
 * the image or costs under 1e9. */
__device__ __forceinline__ int l3d_region_best(const float* cost, int region, int x, int y, int W, int H) {
    const int count = region < 4 ? 7 : 11;
    int chosen = -1;
    float chosen_cost = 1e9f;
    for (int i = 0; i < count; i++) {
        int ox = 0, oy = -3 - 2 * i;
        if (region < 4) l3d_near_offset(i, &ox, &oy);
        int rx, ry;
        l3d_orient(ox, oy, region & 3, &rx, &ry);
        const int qx = x + rx, qy = y + ry;
        if (qx < 0 || qy < 0 || qx >= W || qy >= H) continue;
        const int qi = qy * W + qx;
        const float c = cost[qi];
        if (c < chosen_cost) {
            chosen_cost = c;
            chosen = qi;
        }
    }
    return chosen;
}

/* The best of the eight candidates of a pixel (eight consecutive lanes): the one that a loop over
 * the valid ones in `order`, keeping each that is strictly cheaper than the best so far, would end
 * with.  If one beats *best_cost, *n, *dd and *best_cost become the winner's in all eight lanes. */
__device__ __forceinline__ void l3d_take_best(bool valid, float c, int order, float3 cn, float cd, float3* n,
                                              float* dd, float* best_cost) {
    const bool better = valid && c < *best_cost;
    float m = better ? c : 3.0e38f;
    int key = better ? (order << 8) | (int)(threadIdx.x & 31u) : 0x7fffffff;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, m, off);
        const int ok = __shfl_xor_sync(0xffffffffu, key, off);
        if (om < m || (om == m && ok < key)) {
            m = om;
            key = ok;
        }
    }
    const int from = key & 31;
    const float wx = __shfl_sync(0xffffffffu, cn.x, from), wy = __shfl_sync(0xffffffffu, cn.y, from);
    const float wz = __shfl_sync(0xffffffffu, cn.z, from), wd = __shfl_sync(0xffffffffu, cd, from);
    if (key == 0x7fffffff) return;
    *n = make_float3(wx, wy, wz);
    *dd = wd;
    *best_cost = m;
}

/* One pixel's step by the eight lanes `cand` = 0..7 of a warp, every lane of the warp taking part
 * (`inside` false: it only shuffles).  `s` is prepared; hyp and cost are the view's.  The evaluator
 * gives ray_of, random_normal, random_depth, normalize and cost_of (hypothesis_cost). */
template <class E, class P>
__device__ __forceinline__ void l3d_step_lanes(const E& e, P& s, float4* hyp, float* cost, int x, int y, int W,
                                               int H, bool inside, int cand, float step) {
    const int index = y * W + x;
    const float4 b = inside ? hyp[index] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float3 bn = make_float3(b.x, b.y, b.z);
    float bd = b.w;
    float best_cost = inside ? cost[index] : 0.0f;
    {
        const int chosen = inside ? l3d_region_best(cost, cand, x, y, W, H) : -1;
        bool valid = chosen >= 0;
        float c = 0.0f, dd = 0.0f;
        float3 hn = make_float3(0.0f, 0.0f, 0.0f);
        if (valid) {
            const float4 h = hyp[chosen];
            hn = make_float3(h.x, h.y, h.z);
            const float3 rq = e.ray_of((float)(chosen % W), (float)(chosen / W));
            const float den = e.dot(hn, s.ray);
            dd = e.dot(hn, make_float3(rq.x * h.w, rq.y * h.w, h.w)) / den;
            valid = !(fabsf(den) < 1e-6f);
            if (valid) c = e.cost_of(s, hn, dd);
        }
        l3d_take_best(valid, c, cand, hn, dd, &bn, &bd, &best_cost);
    }
    const float3 view = E::normalize(s.ray);
    const float3 n_random = e.random_normal(s);
    const float d_random = e.random_depth(s);
    const float de = (fmaf(l3d_random(&s.rng), 2.0f, -1.0f) * 0.15f) * step;
    const float d_perturbed = 1.0f / ((1.0f / bd) * (1.0f + de));
    const float r1 = l3d_random(&s.rng), r2 = l3d_random(&s.rng), r3 = l3d_random(&s.rng);
    float3 n_perturbed = E::normalize(make_float3(bn.x + (fmaf(r1, 2.0f, -1.0f) * 0.6f) * step,
                                                  bn.y + (fmaf(r2, 2.0f, -1.0f) * 0.6f) * step,
                                                  bn.z + (fmaf(r3, 2.0f, -1.0f) * 0.6f) * step));
    if (e.dot(n_perturbed, view) >= 0.0f) n_perturbed = bn;
    /* refinement k of the reference's order: (random, random), (perturbed, perturbed), (current,
     * random), (random, current), (current, perturbed), (perturbed, current) normal and depth.  The
     * four at or near the current depth share a hardware quad, the two at the random depth the next:
     * a quad's footprints meet. */
    const int k = cand < 4 ? (0x5431 >> (4 * cand)) & 15 : (cand - 4) * 2;
    const float3 nn = (k == 0 || k == 3) ? n_random : ((k == 1 || k == 5) ? n_perturbed : bn);
    const float dv = (k == 0 || k == 2) ? d_random : ((k == 1 || k == 4) ? d_perturbed : bd);
    const bool valid = inside && cand < 6;
    float c = 0.0f;
    if (valid) c = e.cost_of(s, nn, dv);
    l3d_take_best(valid, c, k, nn, dv, &bn, &bd, &best_cost);
    if (inside && cand == 0) {
        hyp[index] = make_float4(bn.x, bn.y, bn.z, bd);
        cost[index] = best_cost;
    }
}

#endif

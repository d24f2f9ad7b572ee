/*
 * TSDF integration of packed depth maps (frontend/src/app/vision/fusion/tsdf-volume.ts).
 *
 *   k_visible      visibleBricks (tsdf-volume.ts:220-234) on the device: one thread per
 *                  (brick, view) evaluates the reference's FP64 frustum test, in the reference's
 *                  operation order (built with --fmad=false, so no FP64 contraction).
 *   k_integrate    one view per launch (TsdfVolume.integrate, tsdf-volume.ts:240-268).  A thread
 *                  owns four consecutive voxels along x (inside one 8^3 brick): it computes the
 *                  four observations from the L2-resident depth map first (the four depth loads
 *                  in flight together, normals from the decoded-normal table) and touches the
 *                  volume only when one of them updates, with one 128-bit tsdf access and one
 *                  64-bit (Q8.8) or 128-bit (f32) weight access; culled bricks read nothing but
 *                  their mask byte.
 *   k_count_updates
 *                  the visible voxel-views and voxel-updates of a many-view integration, without
 *                  its writes (the algorithmic bytes of the one-view-per-launch form).
 *   k_depth_tiles, k_super_pairs, k_visible_pairs, k_visible_depth
 *                  the depth-aware half of the brick cull (see brick_behind_depths), first for
 *                  blocks of 4^3 bricks, then for the bricks of the blocks not dropped.
 *   k_integrate_many, k_integrate_many_list
 *                  many views per sweep: the same thread keeps its four voxels in registers,
 *                  applies every view in order and writes back once; per-voxel results equal the
 *                  per-view launches bit for bit (the per-voxel update order is unchanged).  The
 *                  list form visits only the bricks some view keeps (k_brick_any, a prefix sum,
 *                  k_brick_list_fill).
 *   k_integrate_list
 *                  one view over the bricks it keeps (k_visible_one_list), grid-stride.
 *
 * Per-voxel arithmetic (tsdf-volume.ts:111-153), fixed order shared with the FP32 restatement:
 *   world = fma(i + 0.5, voxel, origin); cam = R world + t (fma chain); pixel =
 *   rint(fma(f * cam, 1 / cam.z, c)); weight w = max(0.2, |n . normalize(cam)|) x confidence
 *   factor, or the prior weight; tsdf <- fma(tsdf, w0, obs * w) / (w0 + w);
 *   weight <- min(w0 + w, max).  Q8.8 weights: w is rounded to a multiple of 1/256 first, so
 *   weights stay exact integers.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include <cuda_fp16.h>

#include "l3d_fmath.h"
#include "l3d_ieee.h"
#include "l3d_internal.h"

namespace {

__device__ __forceinline__ float dot3f(float3 a, float3 b) {
    return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x));
}
__device__ __forceinline__ float3 normalize3f(float3 v) {
    float il = 1.0f / sqrtf(dot3f(v, v));
    return make_float3(v.x * il, v.y * il, v.z * il);
}
/* normalize3f of a vector whose length lies in [2^-100, 2^100] */
__device__ __forceinline__ float3 normalize_ordinary(float3 v) {
    float il = l3d_rcp_normal(sqrtf(dot3f(v, v)));
    return make_float3(v.x * il, v.y * il, v.z * il);
}
__device__ __forceinline__ float maxw(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float minw(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float clampw(float v, float lo, float hi) { return minw(maxw(v, lo), hi); }

__device__ __forceinline__ float3 unpack_normal(uint32_t packed) {
    float ex = ((float)((packed >> 16) & 63u) / 63.0f) * 2.0f - 1.0f;
    float ey = ((float)((packed >> 22) & 63u) / 63.0f) * 2.0f - 1.0f;
    float3 n = make_float3(ex, ey, (1.0f - fabsf(ex)) - fabsf(ey));
    if (n.z < 0.0f) {
        float sx = n.x >= 0.0f ? 1.0f : -1.0f;
        float sy = n.y >= 0.0f ? 1.0f : -1.0f;
        float nx = (1.0f - fabsf(n.y)) * sx;
        float ny = (1.0f - fabsf(n.x)) * sy;
        n.x = nx;
        n.y = ny;
    }
    return normalize3f(n);
}

/* Observation of one voxel in one view; false when the voxel is not updated. */
__device__ __forceinline__ bool observe(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                        const uint32_t* __restrict__ depth,
                                        const float* __restrict__ prior, int gx, int gy, int gz,
                                        float* obs, float* wout) {
    float wx = fmaf((float)gx + 0.5f, g.voxel, g.origin[0]);
    float wy = fmaf((float)gy + 0.5f, g.voxel, g.origin[1]);
    float wz = fmaf((float)gz + 0.5f, g.voxel, g.origin[2]);
    const float* R = v.R;
    float3 cam = make_float3(fmaf(R[2], wz, fmaf(R[1], wy, fmaf(R[0], wx, v.t[0]))),
                             fmaf(R[5], wz, fmaf(R[4], wy, fmaf(R[3], wx, v.t[1]))),
                             fmaf(R[8], wz, fmaf(R[7], wy, fmaf(R[6], wx, v.t[2]))));
    if (!(cam.z > 0.01f)) return false;
    float iz = 1.0f / cam.z;
    float rx = rintf(fmaf(v.k[0] * cam.x, iz, v.k[2]));
    float ry = rintf(fmaf(v.k[1] * cam.y, iz, v.k[3]));
    if (!(rx >= 0.0f && ry >= 0.0f && rx < (float)v.W && ry < (float)v.H)) return false;
    long long i = (long long)(int)ry * v.W + (int)rx;
    uint32_t packed = __ldg(depth + i);
    float d = l3d_f16_to_f32(packed & 0xffffu);
    float w;
    if (d > 0.0f) {
        float3 n = unpack_normal(packed);
        float3 cn = normalize3f(cam);
        w = maxw(0.2f, fabsf(dot3f(n, cn)));
        if (v.conf > 0.0f) {
            float c = (float)(packed >> 28) / 8.0f;
            float r = clampw(v.conf / d, 0.5f, 2.0f);
            w = w * ((maxw(0.15f, (1.0f - c) * (1.0f - c)) * r) * r);
        }
    } else {
        d = prior ? __ldg(prior + i) : 0.0f;
        w = g.prior_weight;
    }
    if (!(d > 0.0f)) return false;
    float sdf = d - cam.z;
    if (sdf < -g.mu) return false;
    *obs = minw(1.0f, sdf / g.mu);
    *wout = w;
    return true;
}

/* observe() with the same results, reordered for the many-view sweep and split in two.
 * lut_pixel gives the camera point and the depth-map index of every voxel of a quad first, so
 * that their depth loads are in flight together; lut_observe finishes from the loaded sample,
 * with the depth and the truncation test before the weight (most voxels of a view lie behind
 * the surface or outside the truncation band) and the decoded normal from `normals`, a table of
 * unpack_normal over all 4096 normal codes computed with the same arithmetic.  The voxel's world
 * position (fma(i + 0.5, voxel, origin), the same for every view) comes from the caller, and the
 * f16 depth is widened by the hardware conversion, which gives l3d_f16_to_f32's value for every
 * non-NaN half (a NaN fails the d > 0 test either way).
 * ORD: the grid and the view are ordinary (l3d_tsdf_ordinary), so that camera depths, their
 * reciprocals and the divisor mu are normal numbers and pixel indices fit the integer rounding: the
 * same values without the general division's branches and without the conversion pipe, which a voxel
 * and view otherwise enters five times (reciprocal, two roundings, two conversions) at a quarter of
 * the FMA rate or less.  The sweep of 24 views into 512^3: 426 -> 322 us
 * (270 us with bricks handed out, see k_integrate_many_list).  An ordinary map has fewer than 2^31
 * pixels; the indices of any other (17 GB and more with its FP32 depths) have 64 bits. */
template <bool ORD>
using PixelIndex = typename std::conditional<ORD, int, long long>::type;

template <bool ORD>
__device__ __forceinline__ bool lut_pixel(const L3dTsdfView& v, float wx, float wy, float wz,
                                          float3* cam_out, PixelIndex<ORD>* pix) {
    const float* R = v.R;
    float3 cam = make_float3(fmaf(R[2], wz, fmaf(R[1], wy, fmaf(R[0], wx, v.t[0]))),
                             fmaf(R[5], wz, fmaf(R[4], wy, fmaf(R[3], wx, v.t[1]))),
                             fmaf(R[8], wz, fmaf(R[7], wy, fmaf(R[6], wx, v.t[2]))));
    *cam_out = cam;
    if (ORD) {
        const float iz = l3d_rcp_normal(cam.z);
        const unsigned x = l3d_rint_index(fmaf(v.k[0] * cam.x, iz, v.k[2]));
        const unsigned y = l3d_rint_index(fmaf(v.k[1] * cam.y, iz, v.k[3]));
        *pix = (int)(y * (unsigned)v.W + x);
        return cam.z > 0.01f && x < (unsigned)v.W && y < (unsigned)v.H;
    }
    if (!(cam.z > 0.01f)) return false;
    float iz = 1.0f / cam.z;
    float rx = rintf(fmaf(v.k[0] * cam.x, iz, v.k[2]));
    float ry = rintf(fmaf(v.k[1] * cam.y, iz, v.k[3]));
    if (!(rx >= 0.0f && ry >= 0.0f && rx < (float)v.W && ry < (float)v.H)) return false;
    *pix = (PixelIndex<ORD>)(int)ry * v.W + (int)rx;
    return true;
}

template <bool ORD>
__device__ __forceinline__ bool lut_observe(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                            const float* __restrict__ prior,
                                            const float4* __restrict__ normals, float3 cam,
                                            PixelIndex<ORD> i, uint32_t packed, float* obs, float* wout) {
    float d = __half2float(__ushort_as_half((unsigned short)(packed & 0xffffu)));
    const bool stereo = d > 0.0f;
    if (!stereo) d = prior ? __ldg(prior + i) : 0.0f;
    if (!(d > 0.0f)) return false;
    float sdf = d - cam.z;
    if (sdf < -g.mu) return false;
    float w;
    if (stereo) {
        float4 n4 = __ldg(normals + ((packed >> 16) & 4095u));
        float3 cn = ORD ? normalize_ordinary(cam) : normalize3f(cam);
        w = maxw(0.2f, fabsf(dot3f(make_float3(n4.x, n4.y, n4.z), cn)));
        if (v.conf > 0.0f) {
            float c = (float)(packed >> 28) / 8.0f;
            float r = clampw(v.conf / d, 0.5f, 2.0f);
            w = w * ((maxw(0.15f, (1.0f - c) * (1.0f - c)) * r) * r);
        }
    } else {
        w = g.prior_weight;
    }
    /* clipped before the division, an infinite depth (no normal number) gives 1 there too */
    *obs = ORD ? l3d_div_by(fminf(sdf, g.mu), g.mu, g.inv_mu) : minw(1.0f, sdf / g.mu);
    *wout = w;
    return true;
}

__global__ void k_normal_table(float4* normals) {
    const uint32_t code = blockIdx.x * blockDim.x + threadIdx.x;
    if (code >= 4096u) return;
    float3 n = unpack_normal(code << 16);
    normals[code] = make_float4(n.x, n.y, n.z, 0.0f);
}

__device__ __forceinline__ void apply_f32(float& t, float& w0, float obs, float w, float maxw_) {
    t = fmaf(t, w0, obs * w) / (w0 + w);
    w0 = minw(w0 + w, maxw_);
}

__device__ __forceinline__ void apply_q8(float& t, uint32_t& w0i, float obs, float w, unsigned maxq) {
    uint32_t wi = (uint32_t)rintf(w * 256.0f);
    if (wi == 0u) return;
    float w0 = (float)w0i * 0.00390625f;
    float wf = (float)wi * 0.00390625f;
    t = fmaf(t, w0, obs * wf) / (w0 + wf);
    w0i = min(w0i + wi, maxq);
}

/* Voxel coordinates and storage index of the first voxel of quad q (VEC consecutive x).
 * Brick-major order: quad q is quad q % (512 / VEC) of brick q / (512 / VEC), so the 32 threads of a
 * warp stay inside one 8^3 brick (one mask entry, one set of views, converged branches) and touch
 * 32-byte row segments of it; quads of a ragged grid's partial bricks that fall outside the grid are
 * skipped. */
template <int VEC>
__device__ __forceinline__ bool quad_coords(const L3dTsdfGrid& g, const int32_t* coords,
                                            long long q, int* gx, int* gy, int* gz,
                                            long long* idx, long long* brick) {
    if (g.dense) {
        long long b = q / (512 / VEC);
        if (b >= g.bricks) return false;
        int local = (int)(q - b * (512 / VEC)) * VEC;
        /* brick numbers of a dense grid that fits memory fit 32 bits */
        const unsigned bxy = (unsigned)g.nb[0] * (unsigned)g.nb[1];
        const int bz = (int)((unsigned)b / bxy);
        const int rest = (int)((unsigned)b - (unsigned)bz * bxy);
        const int by = rest / g.nb[0], bx = rest - by * g.nb[0];
        *gx = bx * 8 + (local & 7);
        *gy = by * 8 + ((local >> 3) & 7);
        *gz = bz * 8 + (local >> 6);
        if (*gx >= g.dims[0] || *gy >= g.dims[1] || *gz >= g.dims[2]) return false;
        *idx = ((long long)*gz * g.dims[1] + *gy) * g.dims[0] + *gx;
        *brick = b;
    } else {
        long long b = q / (512 / VEC);
        if (b >= g.bricks) return false;
        int local = (int)(q - b * (512 / VEC)) * VEC;
        const int32_t* c = coords + b * 4;
        *gx = c[0] * 8 + (local & 7);
        *gy = c[1] * 8 + ((local >> 3) & 7);
        *gz = c[2] * 8 + (local >> 6);
        *idx = b * 512 + local;
        *brick = b;
    }
    return true;
}

/* Brick coordinates of brick b. */
__device__ __forceinline__ void brick_coords(const L3dTsdfGrid& g, const int32_t* __restrict__ coords, long long b,
                                             int* bx, int* by, int* bz) {
    if (g.dense) {
        *bx = (int)(b % g.nb[0]);
        *by = (int)((b / g.nb[0]) % g.nb[1]);
        *bz = (int)(b / ((long long)g.nb[0] * g.nb[1]));
    } else {
        *bx = coords[b * 4];
        *by = coords[b * 4 + 1];
        *bz = coords[b * 4 + 2];
    }
}

/* visibleBricks (tsdf-volume.ts:220-234) for the brick at (bx, by, bz) and view v, FP64, reference
 * order. */
__device__ __forceinline__ uint8_t brick_visible(const L3dTsdfGrid& g, const L3dTsdfView& v, int bx, int by,
                                                 int bz) {
    double side = g.voxel_d * 8.0;
    double c0 = g.origin_d[0] + (bx + 0.5) * side;
    double c1 = g.origin_d[1] + (by + 0.5) * side;
    double c2 = g.origin_d[2] + (bz + 0.5) * side;
    double radius = g.voxel_d * 8.0 * 0.87 + g.trunc_d;
    const double* R = v.Rd;
    double p0 = R[0] * c0 + R[1] * c1 + R[2] * c2 + v.td[0];
    double p1 = R[3] * c0 + R[4] * c1 + R[5] * c2 + v.td[1];
    double p2 = R[6] * c0 + R[7] * c1 + R[8] * c2 + v.td[2];
    double u = (v.kd[0] * p0) / p2 + v.kd[2];
    double w = (v.kd[1] * p1) / p2 + v.kd[3];
    double z = p2;
    if (z < 0.02 - radius || z > v.max_depth + radius) return 0;
    double margin = (v.kd[0] * radius) / fmax(0.02, z);
    if (u < -margin || w < -margin || u > v.W + margin || w > v.H + margin) return 0;
    return 1;
}

/* The many-view brick mask is brick-major: brick b's flags for views 0..n-1 are the bytes
 * mask[b * mask_stride(n) + v], the row padded with zeros to a multiple of 16 bytes, so a thread
 * reads a brick's views with 128-bit loads. */
__host__ __device__ __forceinline__ int mask_stride(int n_views) { return (n_views + 15) & ~15; }

__global__ void k_visible(const L3dTsdfGrid g, const L3dTsdfView* __restrict__ views, int n_views,
                          const int32_t* __restrict__ coords, uint8_t* __restrict__ mask) {
    const int stride = mask_stride(n_views);
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.bricks * stride) return;
    long long b = t / stride;
    int vi = (int)(t - b * stride);
    int bx, by, bz;
    brick_coords(g, coords, b, &bx, &by, &bz);
    mask[t] = vi < n_views ? brick_visible(g, views[vi], bx, by, bz) : 0;
}

/* The depth-aware half of the brick cull.  A voxel of view v is updated only from the depth d
 * of the pixel it rounds to (the packed map's, or the prior where the map has none), and only
 * if d - z >= -mu for its camera depth z.  The voxel centres of brick b span a box; its eight
 * corners bound every centre's camera depth from below (z is affine) and its pixel to the
 * corners' bounding rectangle widened by a pixel (pixels are rounded to the nearest).  If the
 * smallest corner depth exceeds the largest depth over the depth tiles covering that rectangle
 * by more than mu plus a margin, no voxel of the brick updates: the cull changes which voxels
 * are visited, never a result.  The bound is computed in FP32; the margin (0.2 mm plus 1e-6 of
 * the sum of the magnitudes entering the camera depth, about 17 ulp of it) covers the rounding
 * of this computation and of the kernels' own FP32 camera depth and sdf, and the one-pixel
 * widening covers that of the projections.  Bricks with a corner at z <= 0.02 or a footprint
 * wider than 32 x 32 tiles are kept. */
/* What a box's corners bound: its smallest camera depth and the rectangle of its pixels. */
struct BoxBound {
    float zmin, umin, umax, vmin, vmax;
};
/* Corner c of the box of voxel centres from (lx, ly, lz) to (lx, ly, lz) + span on each axis, whose first
 * corner's camera point is p0; false when the corner is not in front of the camera at an ordinary
 * depth. */
__device__ __forceinline__ bool box_corner(const L3dTsdfView& v, float3 p0, float span, int c, BoxBound* o) {
    const float* R = v.R;
    const float sx = (c & 1) ? span : 0.0f, sy = (c & 2) ? span : 0.0f, sz = (c & 4) ? span : 0.0f;
    const float px = fmaf(R[2], sz, fmaf(R[1], sy, fmaf(R[0], sx, p0.x)));
    const float py = fmaf(R[5], sz, fmaf(R[4], sy, fmaf(R[3], sx, p0.y)));
    const float pz = fmaf(R[8], sz, fmaf(R[7], sy, fmaf(R[6], sx, p0.z)));
    const float iz = l3d_rcp_normal(pz);
    o->zmin = pz;
    o->umin = o->umax = fmaf(v.k[0] * px, iz, v.k[2]);
    o->vmin = o->vmax = fmaf(v.k[1] * py, iz, v.k[3]);
    return pz > 0.02f && pz < 0x1p120f;
}
__device__ __forceinline__ float3 box_origin(const L3dTsdfView& v, float lx, float ly, float lz) {
    const float* R = v.R;
    return make_float3(fmaf(R[2], lz, fmaf(R[1], ly, fmaf(R[0], lx, v.t[0]))),
                       fmaf(R[5], lz, fmaf(R[4], ly, fmaf(R[3], lx, v.t[1]))),
                       fmaf(R[8], lz, fmaf(R[7], ly, fmaf(R[6], lx, v.t[2]))));
}
/* The depth tiles under the bound's pixels: 1 none (nothing projects inside), 0 too many or not
 * numbers (the box is kept), else their rectangle. */
enum TileCover { kTilesKeep, kTilesNone, kTilesRect };
__device__ __forceinline__ TileCover box_tiles(const L3dTsdfView& v, const BoxBound& o, int* tx0, int* tx1, int* ty0,
                                               int* ty1) {
    const float x0 = fmaxf(floorf(o.umin) - 1.0f, 0.0f), x1 = fminf(ceilf(o.umax) + 1.0f, (float)(v.W - 1));
    const float y0 = fmaxf(floorf(o.vmin) - 1.0f, 0.0f), y1 = fminf(ceilf(o.vmax) + 1.0f, (float)(v.H - 1));
    if (!(x1 >= x0) || !(y1 >= y0)) return isnan(x1) || isnan(y1) ? kTilesKeep : kTilesNone;
    *tx0 = (int)x0 / L3D_DEPTH_TILE;
    *tx1 = (int)x1 / L3D_DEPTH_TILE;
    *ty0 = (int)y0 / L3D_DEPTH_TILE;
    *ty1 = (int)y1 / L3D_DEPTH_TILE;
    return *tx1 - *tx0 >= 32 || *ty1 - *ty0 >= 32 ? kTilesKeep : kTilesRect;
}
__device__ __forceinline__ bool box_behind(const L3dTsdfGrid& g, const L3dTsdfView& v, float lx, float ly, float lz,
                                           float span, float zmin, float dmax) {
    const float mag = fabsf(lx) + fabsf(ly) + fabsf(lz) + 3.0f * span + fabsf(v.t[0]) + fabsf(v.t[1]) + fabsf(v.t[2]);
    return zmin - dmax > g.mu + 2e-4f + 1e-6f * (mag + dmax);
}

/* brick_behind_depths for the axis-aligned box of voxel centres from (lx, ly, lz) to
 * (lx, ly, lz) + span on each axis. */
__device__ __forceinline__ bool box_behind_depths(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                                  const float* __restrict__ tiles, float lx, float ly,
                                                  float lz, float span) {
    const float3 p0 = box_origin(v, lx, ly, lz);
    BoxBound o = {3e38f, 3e38f, -3e38f, 3e38f, -3e38f};
#pragma unroll
    for (int c = 0; c < 8; c++) {
        BoxBound k;
        if (!box_corner(v, p0, span, c, &k)) return false;
        o.zmin = fminf(o.zmin, k.zmin);
        o.umin = fminf(o.umin, k.umin);
        o.umax = fmaxf(o.umax, k.umax);
        o.vmin = fminf(o.vmin, k.vmin);
        o.vmax = fmaxf(o.vmax, k.vmax);
    }
    int tx0, tx1, ty0, ty1;
    const TileCover cover = box_tiles(v, o, &tx0, &tx1, &ty0, &ty1);
    if (cover != kTilesRect) return cover == kTilesNone;
    const int tw = (v.W + L3D_DEPTH_TILE - 1) / L3D_DEPTH_TILE;
    const float* vt = tiles + v.tile_off;
    float dmax = 0.0f;
    for (int ty = ty0; ty <= ty1; ty++)
        for (int tx = tx0; tx <= tx1; tx++) dmax = fmaxf(dmax, __ldg(vt + (long long)ty * tw + tx));
    return box_behind(g, v, lx, ly, lz, span, o.zmin, dmax);
}

/* The same by eight consecutive lanes (every lane of the warp taking part), a corner and an eighth of the
 * tiles each, for launches of too few boxes to hide one thread's chain of corners and tile loads; the
 * same answer in all eight. */
__device__ __forceinline__ bool box_behind_depths_lanes(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                                        const float* __restrict__ tiles, float lx, float ly,
                                                        float lz, float span) {
    const int lane = threadIdx.x & 31, c = lane & 7;
    BoxBound o;
    const bool bad = !box_corner(v, box_origin(v, lx, ly, lz), span, c, &o);
    const bool keep = (__ballot_sync(0xffffffffu, bad) >> (lane & 24) & 255u) != 0u;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
        o.zmin = fminf(o.zmin, __shfl_xor_sync(0xffffffffu, o.zmin, off));
        o.umin = fminf(o.umin, __shfl_xor_sync(0xffffffffu, o.umin, off));
        o.umax = fmaxf(o.umax, __shfl_xor_sync(0xffffffffu, o.umax, off));
        o.vmin = fminf(o.vmin, __shfl_xor_sync(0xffffffffu, o.vmin, off));
        o.vmax = fmaxf(o.vmax, __shfl_xor_sync(0xffffffffu, o.vmax, off));
    }
    int tx0 = 0, tx1 = 0, ty0 = 0, ty1 = 0;
    const TileCover cover = keep ? kTilesKeep : box_tiles(v, o, &tx0, &tx1, &ty0, &ty1);
    float dmax = 0.0f;
    if (cover == kTilesRect) {
        const int tw = (v.W + L3D_DEPTH_TILE - 1) / L3D_DEPTH_TILE, n = tx1 - tx0 + 1, count = n * (ty1 - ty0 + 1);
        const float* vt = tiles + v.tile_off;
        for (int i = c; i < count; i += 8) {
            const int row = i / n;
            dmax = fmaxf(dmax, __ldg(vt + (long long)(ty0 + row) * tw + tx0 + (i - row * n)));
        }
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, off));
    return cover == kTilesNone || (cover == kTilesRect && box_behind(g, v, lx, ly, lz, span, o.zmin, dmax));
}

template <bool LANES>
__device__ __forceinline__ bool brick_behind_depths(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                                    const float* __restrict__ tiles, int bx, int by, int bz) {
    const float lx = fmaf((float)(bx * 8) + 0.5f, g.voxel, g.origin[0]);
    const float ly = fmaf((float)(by * 8) + 0.5f, g.voxel, g.origin[1]);
    const float lz = fmaf((float)(bz * 8) + 0.5f, g.voxel, g.origin[2]);
    return LANES ? box_behind_depths_lanes(g, v, tiles, lx, ly, lz, 7.0f * g.voxel)
                 : box_behind_depths(g, v, tiles, lx, ly, lz, 7.0f * g.voxel);
}

/* Depth tiles of view v (see l3d_launch_depth_tiles): thread t takes row t % 8 of tile t / 8
 * (eight pixels), and the eight threads of a tile, consecutive lanes of one warp, combine their
 * maxima with shuffles; lane 0 of the group writes the tile. */
__device__ __forceinline__ void depth_tile(const L3dTsdfView& v, const uint32_t* __restrict__ depth,
                                           const float* __restrict__ prior, float* __restrict__ tiles,
                                           long long t) {
    static_assert(L3D_DEPTH_TILE == 8, "eight rows per tile, eight lanes per tile");
    const int tw = (v.W + L3D_DEPTH_TILE - 1) / L3D_DEPTH_TILE, th = (v.H + L3D_DEPTH_TILE - 1) / L3D_DEPTH_TILE;
    const long long tile = t >> 3;
    const int row = (int)(t & 7);
    float m = 0.0f;
    if (tile < (long long)tw * th) {
        const int tx = (int)(tile % tw), ty = (int)(tile / tw);
        const int y = ty * L3D_DEPTH_TILE + row;
        if (y < v.H)
            for (int x = tx * L3D_DEPTH_TILE; x < min(v.W, (tx + 1) * L3D_DEPTH_TILE); x++) {
                const long long i = (long long)y * v.W + x;
                float d = __half2float(__ushort_as_half((unsigned short)(__ldg(depth + i) & 0xffffu)));
                if (!(d > 0.0f)) d = prior ? __ldg(prior + i) : 0.0f;
                if (d > m) m = d;  /* NaN never raises the maximum: such a pixel never updates */
            }
    }
    /* the tile's eight lanes are aligned groups of a warp (blocks are whole warps) */
    for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (row == 0 && tile < (long long)tw * th) tiles[v.tile_off + tile] = m;
}

__global__ void k_depth_tiles(const L3dTsdfView* __restrict__ views, int n_views,
                              const uint32_t* const* __restrict__ depths, const float* __restrict__ priors,
                              float* __restrict__ tiles, long long max_tiles) {
    const int vi = blockIdx.y;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;  /* every lane takes part */
    const L3dTsdfView& v = views[vi];
    depth_tile(v, depths[vi], v.has_prior ? priors + v.prior_off : nullptr, tiles, t);
}

__global__ void k_depth_tiles_one(const L3dTsdfView v, const uint32_t* __restrict__ depth,
                                  const float* __restrict__ prior, float* __restrict__ tiles, int32_t* list) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *list = 0;  /* the next launch appends to it */
    depth_tile(v, depth, v.has_prior ? prior : nullptr, tiles, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

/* Super-bricks of a dense grid: blocks of L3D_SUPER^3 bricks.  A super-brick whose voxel centres (the
 * grid's edge cut off) are behind view v's depths by the test of brick_behind_depths holds only bricks
 * that are; the others are listed with their view, and only their bricks are tested one by one
 * (k_visible_pairs), 64 to a pair, a warp's lanes at one view and one place.  24 views and 512^3 voxels: a
 * thread per (brick, view) that looked its super-brick's flag up took 162 us with the flags, these two
 * take 55. */
constexpr int L3D_SUPER = 4;
__host__ __device__ __forceinline__ int super_count(const L3dTsdfGrid& g, int axis) {
    return (g.nb[axis] + L3D_SUPER - 1) / L3D_SUPER;
}

/* pairs[0] counts the kept pairs (zeroed), pairs[1 ..] receives super-brick * n_views + view in any order;
 * eight lanes per pair. */
__global__ void __launch_bounds__(256) k_super_pairs(const L3dTsdfGrid g, const L3dTsdfView* __restrict__ views,
                                                     int n_views, const float* __restrict__ tiles,
                                                     uint32_t* __restrict__ pairs) {
    const long long n = (long long)super_count(g, 0) * super_count(g, 1) * super_count(g, 2) * n_views;
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const long long p = t < n ? t : n - 1;  /* every lane takes part */
    const long long sb = p / n_views;
    const int vi = (int)(p - sb * n_views);
    const int sx = (int)(sb % super_count(g, 0));
    const int sy = (int)((sb / super_count(g, 0)) % super_count(g, 1));
    const int sz = (int)(sb / ((long long)super_count(g, 0) * super_count(g, 1)));
    constexpr int V = 8 * L3D_SUPER;
    /* the box's far corner: the last voxel of the super-brick inside the grid on each axis */
    const int ex = min(V, g.dims[0] - sx * V) - 1, ey = min(V, g.dims[1] - sy * V) - 1;
    const int ez = min(V, g.dims[2] - sz * V) - 1;
    const int e = max(ex, max(ey, ez));
    const bool behind = box_behind_depths_lanes(g, views[vi], tiles, fmaf((float)(sx * V) + 0.5f, g.voxel, g.origin[0]),
                                                fmaf((float)(sy * V) + 0.5f, g.voxel, g.origin[1]),
                                                fmaf((float)(sz * V) + 0.5f, g.voxel, g.origin[2]), (float)e * g.voxel);
    const bool put = t < n && !behind && (threadIdx.x & 7) == 0;
    const unsigned who = __ballot_sync(0xffffffffu, put);
    if (!who) return;
    const int lane = threadIdx.x & 31, first = __ffs(who) - 1;
    uint32_t at = 0;
    if (lane == first) at = atomicAdd(pairs, (uint32_t)__popc(who));
    at = __shfl_sync(0xffffffffu, at, first);
    if (put) pairs[1 + at + __popc(who & ((1u << lane) - 1u))] = (uint32_t)p;
}

/* The mask bytes of the listed super-bricks' bricks (the mask was zeroed), a thread per brick. */
__global__ void __launch_bounds__(256) k_visible_pairs(const L3dTsdfGrid g, const L3dTsdfView* __restrict__ views,
                                                       int n_views, const float* __restrict__ tiles,
                                                       const uint32_t* __restrict__ pairs, uint8_t* __restrict__ mask) {
    constexpr int PER = L3D_SUPER * L3D_SUPER * L3D_SUPER;
    const int stride = mask_stride(n_views);
    const long long n = (long long)__ldg(pairs) * PER;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const uint32_t p = __ldg(pairs + 1 + i / PER);
        const int sb = (int)(p / (uint32_t)n_views), vi = (int)(p - (uint32_t)sb * n_views), k = (int)(i % PER);
        const int bx = sb % super_count(g, 0) * L3D_SUPER + k % L3D_SUPER;
        const int by = sb / super_count(g, 0) % super_count(g, 1) * L3D_SUPER + k / L3D_SUPER % L3D_SUPER;
        const int bz = sb / (super_count(g, 0) * super_count(g, 1)) * L3D_SUPER + k / (L3D_SUPER * L3D_SUPER);
        if (bx >= g.nb[0] || by >= g.nb[1] || bz >= g.nb[2]) continue;
        const L3dTsdfView& v = views[vi];
        /* a brick behind the depths needs no frustum test: it is dropped either way */
        if (!brick_behind_depths<false>(g, v, tiles, bx, by, bz) && brick_visible(g, v, bx, by, bz))
            mask[(((long long)bz * g.nb[1] + by) * g.nb[0] + bx) * stride + vi] = 1;
    }
}

/* The whole mask, a thread per (brick, view): brick pools. */
__global__ void k_visible_depth(const L3dTsdfGrid g, const L3dTsdfView* __restrict__ views, int n_views,
                                const int32_t* __restrict__ coords, const float* __restrict__ tiles,
                                uint8_t* __restrict__ mask) {
    const int stride = mask_stride(n_views);
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.bricks * stride) return;
    long long b = t / stride;
    int vi = (int)(t - b * stride);
    if (vi >= n_views) {
        mask[t] = 0;
        return;
    }
    int bx, by, bz;
    brick_coords(g, coords, b, &bx, &by, &bz);
    mask[t] = brick_behind_depths<false>(g, views[vi], tiles, bx, by, bz) ? 0 : brick_visible(g, views[vi], bx, by, bz);
}

/* The kept bricks of one view, a thread per brick, or eight (LANES): list[0] counts them (zeroed before the
 * launch), list[1..] receives their indices in any order.  Eight lanes shorten the walk over a brick's tiles,
 * one makes an eighth of the frustum tests' FP64 instructions: a view of 640x480 and all its launches take
 * 24.8 against 41.7 us at 3472 bricks, 25.6 against 29.9 at 110592, but 32.4 against 31.1 at 175616 and
 * 39.8 against 32.4 at 262144. */
constexpr long long LANES_BRICKS = 1 << 17;
template <bool LANES>
__global__ void __launch_bounds__(128) k_visible_one_list(const L3dTsdfGrid g, const L3dTsdfView v,
                                                          const int32_t* __restrict__ coords,
                                                          const float* __restrict__ tiles, int32_t* __restrict__ list) {
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> (LANES ? 3 : 0);
    const long long b = t < g.bricks ? t : g.bricks - 1;  /* every lane takes part */
    int bx, by, bz;
    brick_coords(g, coords, b, &bx, &by, &bz);
    const bool behind = brick_behind_depths<LANES>(g, v, tiles, bx, by, bz);
    if (behind || t >= g.bricks || (LANES && (threadIdx.x & 7) != 0) || !brick_visible(g, v, bx, by, bz)) return;
    list[1 + atomicAdd(list, 1)] = (int32_t)b;
}

__global__ void k_visible_one(const L3dTsdfGrid g, const L3dTsdfView v,
                              const int32_t* __restrict__ coords, uint8_t* __restrict__ mask) {
    long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= g.bricks) return;
    int bx, by, bz;
    brick_coords(g, coords, b, &bx, &by, &bz);
    mask[b] = brick_visible(g, v, bx, by, bz);
}

/* One view per launch.  LUT: the normal of a depth sample comes from the 4096-entry normal
 * table and a quad's four depth loads are issued together (lut_pixel / lut_observe, the sweep's
 * path, equal to observe() bit for bit); otherwise observe() decodes each normal. */
template <int VEC, bool Q8, bool LUT, bool ORD>
__device__ __forceinline__ void integrate_quad(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                               const int32_t* __restrict__ coords,
                                               const uint8_t* __restrict__ mask,
                                               const uint32_t* __restrict__ depth,
                                               const float* __restrict__ prior,
                                               const float4* __restrict__ normals,
                                               float* __restrict__ tsdf, void* __restrict__ weight,
                                               long long q) {
    int gx, gy, gz;
    long long idx, brick;
    if (!quad_coords<VEC>(g, coords, q, &gx, &gy, &gz, &idx, &brick)) return;
    if (mask && !mask[brick]) return;
    float obs[VEC], w[VEC];
    bool ok[VEC];
    bool any = false;
    if (LUT) {
        const float wy = fmaf((float)gy + 0.5f, g.voxel, g.origin[1]);
        const float wz = fmaf((float)gz + 0.5f, g.voxel, g.origin[2]);
        const float* pr = v.has_prior ? prior : nullptr;
        float3 cam[VEC];
        PixelIndex<ORD> pix[VEC];
        uint32_t packed[VEC];
#pragma unroll
        for (int j = 0; j < VEC; j++)
            ok[j] = lut_pixel<ORD>(v, fmaf((float)(gx + j) + 0.5f, g.voxel, g.origin[0]), wy, wz, &cam[j], &pix[j]);
#pragma unroll
        for (int j = 0; j < VEC; j++) packed[j] = ok[j] ? __ldg(depth + pix[j]) : 0u;
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            ok[j] = ok[j] && lut_observe<ORD>(g, v, pr, normals, cam[j], pix[j], packed[j], &obs[j], &w[j]);
            any |= ok[j];
        }
    } else {
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            ok[j] = observe(g, v, depth, v.has_prior ? prior : nullptr, gx + j, gy, gz, &obs[j], &w[j]);
            any |= ok[j];
        }
    }
    if (!any) return;
    if (VEC == 4) {
        float4 t4 = *(const float4*)(tsdf + idx);
        float t[4] = {t4.x, t4.y, t4.z, t4.w};
        if (Q8) {
            ushort4 w4 = *(const ushort4*)((const uint16_t*)weight + idx);
            uint32_t wq[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (ok[j]) apply_q8(t[j], wq[j], obs[j], w[j], g.max_q);
            *(ushort4*)((uint16_t*)weight + idx) =
                make_ushort4((uint16_t)wq[0], (uint16_t)wq[1], (uint16_t)wq[2], (uint16_t)wq[3]);
        } else {
            float4 w4 = *(const float4*)((const float*)weight + idx);
            float ww[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (ok[j]) apply_f32(t[j], ww[j], obs[j], w[j], g.max_weight);
            *(float4*)((float*)weight + idx) = make_float4(ww[0], ww[1], ww[2], ww[3]);
        }
        *(float4*)(tsdf + idx) = make_float4(t[0], t[1], t[2], t[3]);
    } else {
        float t = tsdf[idx];
        if (Q8) {
            uint32_t wq = ((const uint16_t*)weight)[idx];
            apply_q8(t, wq, obs[0], w[0], g.max_q);
            ((uint16_t*)weight)[idx] = (uint16_t)wq;
        } else {
            float ww = ((const float*)weight)[idx];
            apply_f32(t, ww, obs[0], w[0], g.max_weight);
            ((float*)weight)[idx] = ww;
        }
        tsdf[idx] = t;
    }
}

template <int VEC, bool Q8, bool LUT>
__global__ void __launch_bounds__(256) k_integrate(const L3dTsdfGrid g, const L3dTsdfView v,
                                                   const int32_t* __restrict__ coords,
                                                   const uint8_t* __restrict__ mask,
                                                   const uint32_t* __restrict__ depth,
                                                   const float* __restrict__ prior,
                                                   const float4* __restrict__ normals,
                                                   float* __restrict__ tsdf, void* __restrict__ weight,
                                                   long long quads) {
    long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= quads) return;
    integrate_quad<VEC, Q8, LUT, false>(g, v, coords, mask, depth, prior, normals, tsdf, weight, q);
}

/* One view over its kept bricks only: list[0] bricks listed at list[1..] (by
 * k_visible_one_list, in any order; each brick's voxels are updated independently), a
 * grid-stride loop over their quads. */
template <int VEC, bool Q8>
__global__ void __launch_bounds__(256) k_integrate_list(const L3dTsdfGrid g, const L3dTsdfView v,
                                                        const int32_t* __restrict__ coords,
                                                        const int32_t* __restrict__ list,
                                                        const uint32_t* __restrict__ depth,
                                                        const float* __restrict__ prior,
                                                        const float4* __restrict__ normals,
                                                        float* __restrict__ tsdf,
                                                        void* __restrict__ weight) {
    constexpr int PER = 512 / VEC;
    const long long n = (long long)__ldg(list) * PER;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const long long b = __ldg(list + 1 + i / PER);
        integrate_quad<VEC, Q8, true, true>(g, v, coords, nullptr, depth, prior, normals, tsdf, weight,
                                      b * PER + i % PER);
    }
}

/* One quad of the many-view sweep: its voxels stay in registers while every view that keeps
 * its brick is applied in view order; written back once. */
template <int VEC, bool Q8, bool ORD>
__device__ __forceinline__ void sweep_quad(const L3dTsdfGrid& g, const L3dTsdfView* __restrict__ views,
                                           int n_views, const int32_t* __restrict__ coords,
                                           const uint8_t* __restrict__ mask,
                                           const uint32_t* const* __restrict__ depths,
                                           const float* __restrict__ priors,
                                           const float4* __restrict__ normals,
                                           float* __restrict__ tsdf, void* __restrict__ weight,
                                           long long q) {
    int gx, gy, gz;
    long long idx, brick;
    if (!quad_coords<VEC>(g, coords, q, &gx, &gy, &gz, &idx, &brick)) return;
    /* the brick's row of the mask, 16 views per 128-bit load; a brick no view keeps is left
     * without touching the volume */
    const int stride = mask_stride(n_views);
    const uint4* mrow = (const uint4*)(mask + brick * stride);
    uint32_t any = 0u;
    for (int k = 0; k < stride / 16; k++) {
        const uint4 m = __ldg(mrow + k);
        any |= m.x | m.y | m.z | m.w;
    }
    if (!any) return;
    float t[VEC];
    float wf[VEC];
    uint32_t wq[VEC];
    float wx[VEC];
#pragma unroll
    for (int j = 0; j < VEC; j++) wx[j] = fmaf((float)(gx + j) + 0.5f, g.voxel, g.origin[0]);
    const float wy = fmaf((float)gy + 0.5f, g.voxel, g.origin[1]);
    const float wz = fmaf((float)gz + 0.5f, g.voxel, g.origin[2]);
    /* the quad's volume values are loaded up front (one 128-bit tsdf load, one 64-bit Q8.8 or
     * 128-bit f32 weight load), so their latency overlaps the first view's projection; they are
     * written back only when a view updated them */
    if (VEC == 4) {
        const float4 t4 = *(const float4*)(tsdf + idx);
        t[0] = t4.x; t[1] = t4.y; t[2] = t4.z; t[3] = t4.w;
        if (Q8) {
            const ushort4 w4 = *(const ushort4*)((const uint16_t*)weight + idx);
            wq[0] = w4.x; wq[1] = w4.y; wq[2] = w4.z; wq[3] = w4.w;
        } else {
            const float4 w4 = *(const float4*)((const float*)weight + idx);
            wf[0] = w4.x; wf[1] = w4.y; wf[2] = w4.z; wf[3] = w4.w;
        }
    } else {
        t[0] = tsdf[idx];
        if (Q8) wq[0] = ((const uint16_t*)weight)[idx];
        else wf[0] = ((const float*)weight)[idx];
    }
    bool loaded = false;
    /* the views that keep the brick, 16 at a time, in view order: a mask byte is 0 or 1, so
     * (word * 0x10204080) >> 28 gathers a 32-bit word's four flags into four bits */
    for (int w0 = 0; w0 < n_views; w0 += 16) {
      const uint4 m = __ldg(mrow + w0 / 16);
      uint32_t seen = ((m.x * 0x10204080u) >> 28) | (((m.y * 0x10204080u) >> 28) << 4) |
                      (((m.z * 0x10204080u) >> 28) << 8) | (((m.w * 0x10204080u) >> 28) << 12);
      while (seen) {
        const int vi = w0 + __ffs(seen) - 1;
        seen &= seen - 1u;
        const L3dTsdfView& v = views[vi];
        const uint32_t* depth = depths[vi];
        const float* prior = v.has_prior ? priors + v.prior_off : nullptr;
        float3 cam[VEC];
        PixelIndex<ORD> pix[VEC];
        bool in[VEC];
        uint32_t packed[VEC];
#pragma unroll
        for (int j = 0; j < VEC; j++) in[j] = lut_pixel<ORD>(v, wx[j], wy, wz, &cam[j], &pix[j]);
#pragma unroll
        for (int j = 0; j < VEC; j++) packed[j] = in[j] ? __ldg(depth + pix[j]) : 0u;
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            float obs, w;
            if (!in[j] || !lut_observe<ORD>(g, v, prior, normals, cam[j], pix[j], packed[j], &obs, &w)) continue;
            loaded = true;
            if (Q8) apply_q8(t[j], wq[j], obs, w, g.max_q);
            else apply_f32(t[j], wf[j], obs, w, g.max_weight);
        }
      }
    }
    if (!loaded) return;
    if (VEC == 4) {
        *(float4*)(tsdf + idx) = make_float4(t[0], t[1], t[2], t[3]);
        if (Q8)
            *(ushort4*)((uint16_t*)weight + idx) =
                make_ushort4((uint16_t)wq[0], (uint16_t)wq[1], (uint16_t)wq[2], (uint16_t)wq[3]);
        else
            *(float4*)((float*)weight + idx) = make_float4(wf[0], wf[1], wf[2], wf[3]);
    } else {
        tsdf[idx] = t[0];
        if (Q8) ((uint16_t*)weight)[idx] = (uint16_t)wq[0];
        else ((float*)weight)[idx] = wf[0];
    }
}

template <int VEC, bool Q8>
__global__ void __launch_bounds__(256, 4) k_integrate_many(const L3dTsdfGrid g,
                                                        const L3dTsdfView* __restrict__ views,
                                                        int n_views,
                                                        const int32_t* __restrict__ coords,
                                                        const uint8_t* __restrict__ mask,
                                                        const uint32_t* const* __restrict__ depths,
                                                        const float* __restrict__ priors,
                                                        const float4* __restrict__ normals,
                                                        float* __restrict__ tsdf,
                                                        void* __restrict__ weight,
                                                        long long q_begin, long long q_end) {
    const long long q = q_begin + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= q_end) return;
    sweep_quad<VEC, Q8, false>(g, views, n_views, coords, mask, depths, priors, normals, tsdf, weight, q);
}

/* Passes per warp up to which the sweep's warps stride through them by their numbers: asking costs a round
 * trip each and the counter's clearing a node of the stream (66^3, 5 views of 320x240: 86.7 us with
 * asking, 84.4 without), and balances nothing yet; at 8 rounds it would (256^3, 24 views: 171.6 against
 * 197.8). */
constexpr uint32_t kFixedRounds = 3;

/* The sweep over the bricks some view keeps: list holds them in ascending order
 * (l3d_launch_tsdf_brick_list), prefix[b] is the number of kept bricks below brick b, so the
 * kept bricks of [b_begin, b_end) are list[prefix[b_begin] .. prefix[b_end]).  A warp's pass takes 32
 * quads of a brick.  Every warp starts with a share of passes by its number and, beyond kFixedRounds,
 * takes the next ones from *next (zeroed before the launch) until none is left: bricks cost as much as
 * views keep them, and a fixed share for each warp leaves warps idle at the end (24 views into 512^3: 322
 * us, handed out 270 us).  A share is at most a brick, for few atomics, and an eighth of what there is for
 * each warp, at least a pass: whole bricks left most of the chip waiting for warps that walked their 4
 * or 16 passes alone where few bricks are kept (host call, 24 views of 320x240: 101^3 278 -> 147 us, 256^3
 * 236 -> 171).  Each quad is still one thread's, so results equal k_integrate_many's. */
template <int VEC, bool Q8>
__global__ void __launch_bounds__(256, 4) k_integrate_many_list(const L3dTsdfGrid g,
                                                             const L3dTsdfView* __restrict__ views,
                                                             int n_views,
                                                             const int32_t* __restrict__ coords,
                                                             const uint8_t* __restrict__ mask,
                                                             const uint32_t* const* __restrict__ depths,
                                                             const float* __restrict__ priors,
                                                             const float4* __restrict__ normals,
                                                             float* __restrict__ tsdf,
                                                             void* __restrict__ weight,
                                                             const uint32_t* __restrict__ prefix,
                                                             const int32_t* __restrict__ list,
                                                             uint32_t* __restrict__ next,
                                                             long long b_begin, long long b_end) {
    constexpr int PER = 512 / VEC;
    /* the view table in shared memory, copied once per block */
    extern __shared__ __align__(16) unsigned char sweep_smem[];
    L3dTsdfView* sv = reinterpret_cast<L3dTsdfView*>(sweep_smem);
    {
        const int words = n_views * (int)(sizeof(L3dTsdfView) / 8);
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(views);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(sweep_smem);
        for (int k = threadIdx.x; k < words; k += blockDim.x) dst[k] = __ldg(src + k);
        __syncthreads();
    }
    constexpr uint32_t PASSES = PER / 32;  /* of a warp over a brick */
    const uint32_t first = __ldg(prefix + b_begin), passes = (__ldg(prefix + b_end) - first) * PASSES;
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t share = min(max(passes / (warps * 8u), 1u), PASSES);
    const bool fixed = passes <= warps * kFixedRounds;
    uint32_t at = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    for (;;) {
        const uint32_t begin = at * share, end = min(begin + share, passes);
        for (uint32_t i = begin; i < end; i++) {
            const long long b = __ldg(list + first + i / PASSES);
            sweep_quad<VEC, Q8, true>(g, sv, n_views, coords, mask, depths, priors, normals, tsdf, weight,
                                      b * PER + (i % PASSES) * 32u + lane);
            __syncwarp();
        }
        if (fixed) {
            at += warps;
        } else {
            if (lane == 0) at = atomicAdd(next, 1u);
            at = warps + __shfl_sync(0xffffffffu, at, 0);
        }
        if (at * share >= passes) return;
    }
}
static_assert(sizeof(L3dTsdfView) % 8 == 0, "the view table is copied in 8-byte words");

/* flags[b] = 1 if some view keeps brick b (its mask row is not all zero), for b < bricks;
 * flags[bricks] = 0, so that an exclusive scan of bricks + 1 flags ends with the total. */
__global__ void k_brick_any(const uint8_t* __restrict__ mask, int stride, long long bricks,
                            uint32_t* __restrict__ flags) {
    const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (b > bricks) return;
    uint32_t any = 0u;
    if (b < bricks) {
        const uint4* row = (const uint4*)(mask + b * stride);
        for (int k = 0; k < stride / 16; k++) {
            const uint4 m = __ldg(row + k);
            any |= m.x | m.y | m.z | m.w;
        }
    }
    flags[b] = any ? 1u : 0u;
}

__global__ void k_brick_list_fill(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ prefix,
                                  long long bricks, int32_t* __restrict__ list) {
    const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (b < bricks && flags[b]) list[prefix[b]] = (int32_t)b;
}

/* The work of a many-view integration without its writes: per voxel, the views whose brick
 * culling keeps it (visible) and the views that update it (lut_observe true), summed over the
 * volume into counts[0] (visible voxel-views) and counts[1] (voxel-updates). */
template <int VEC>
__global__ void __launch_bounds__(256) k_count_updates(const L3dTsdfGrid g,
                                                       const L3dTsdfView* __restrict__ views,
                                                       int n_views, const int32_t* __restrict__ coords,
                                                       const uint8_t* __restrict__ mask,
                                                       const uint32_t* const* __restrict__ depths,
                                                       const float* __restrict__ priors,
                                                       const float4* __restrict__ normals,
                                                       long long quads,
                                                       unsigned long long* __restrict__ counts) {
    long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long vis = 0, upd = 0;
    int gx, gy, gz;
    long long idx, brick;
    if (q < quads && quad_coords<VEC>(g, coords, q, &gx, &gy, &gz, &idx, &brick)) {
        const float wy = fmaf((float)gy + 0.5f, g.voxel, g.origin[1]);
        const float wz = fmaf((float)gz + 0.5f, g.voxel, g.origin[2]);
        for (int vi = 0; vi < n_views; vi++) {
            if (!mask[brick * mask_stride(n_views) + vi]) continue;
            vis += VEC;
            const L3dTsdfView& v = views[vi];
            const float* prior = v.has_prior ? priors + v.prior_off : nullptr;
#pragma unroll
            for (int j = 0; j < VEC; j++) {
                float3 cam;
                PixelIndex<false> pix;
                float obs, w;
                if (lut_pixel<false>(v, fmaf((float)(gx + j) + 0.5f, g.voxel, g.origin[0]), wy, wz, &cam, &pix) &&
                    lut_observe<false>(g, v, prior, normals, cam, pix, __ldg(depths[vi] + pix), &obs, &w))
                    upd++;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        vis += __shfl_down_sync(0xffffffffu, vis, o);
        upd += __shfl_down_sync(0xffffffffu, upd, o);
    }
    if ((threadIdx.x & 31) == 0 && (vis || upd)) {
        atomicAdd(counts, vis);
        atomicAdd(counts + 1, upd);
    }
}

/* ---- differentiable integration: depth from an FP32 map ---- */

/* lut_pixel and lut_observe with the stereo depth read from an FP32 map (validity, normal and cost still
 * come from the packed map), plus the derivatives of the observation and of its weight with respect
 * to that depth.  *pix is the map index whose depth was used, or -1 for a prior observation
 * (which does not depend on the map).  With depthf[i] == unpack_depth(packed[i]) the results
 * equal observe()'s bit for bit. */
template <bool ORD>
__device__ __forceinline__ bool observe_diff(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                             const float* __restrict__ depthf,
                                             const float* __restrict__ prior,
                                             const float4* __restrict__ normals, float3 cam, uint32_t packed,
                                             PixelIndex<ORD>* pix, float* obs, float* wout, float* dobs,
                                             float* dw) {
    const PixelIndex<ORD> i = *pix;
    const bool stereo = __half2float(__ushort_as_half((unsigned short)(packed & 0xffffu))) > 0.0f;
    const float d = stereo ? __ldg(depthf + i) : (prior ? __ldg(prior + i) : 0.0f);
    if (!(d > 0.0f)) return false;
    const float sdf = d - cam.z;
    if (sdf < -g.mu) return false;
    float w = g.prior_weight, dwdd = 0.0f;
    if (stereo) {
        const float4 n4 = __ldg(normals + ((packed >> 16) & 4095u));
        const float3 cn = ORD ? normalize_ordinary(cam) : normalize3f(cam);
        w = maxw(0.2f, fabsf(dot3f(make_float3(n4.x, n4.y, n4.z), cn)));
        if (v.conf > 0.0f) {
            const float c = (float)(packed >> 28) / 8.0f;
            const float q = v.conf / d;
            const float r = clampw(q, 0.5f, 2.0f);
            const float m = maxw(0.15f, (1.0f - c) * (1.0f - c));
            /* w m r^2 with r = conf / d inside the clamp: dr/dd = -conf / d^2 = -r / d */
            if (q > 0.5f && q < 2.0f) dwdd = w * m * 2.0f * r * (-q / d);
            w = w * ((m * r) * r);
        }
    } else {
        *pix = -1;
    }
    /* past the truncation the observation is the constant 1 (an infinite depth included) */
    const bool past = sdf > g.mu;
    *obs = ORD ? (past ? 1.0f : l3d_div_by(sdf, g.mu, g.inv_mu)) : minw(1.0f, sdf / g.mu);
    *dobs = past ? 0.0f : (ORD ? g.inv_mu : 1.0f / g.mu);
    *wout = w;
    *dw = dwdd;
    return true;
}

/* The pixels and packed samples of a quad of VEC voxels along x (brick-major order): bit j of the result
 * is set where voxel j projects into the map. */
template <int VEC, bool ORD>
__device__ __forceinline__ unsigned quad_pixels(const L3dTsdfGrid& g, const L3dTsdfView& v,
                                                const uint32_t* __restrict__ depth, int gx, int gy, int gz,
                                                float3* cam, PixelIndex<ORD>* pix, uint32_t* packed) {
    const float wy = fmaf((float)gy + 0.5f, g.voxel, g.origin[1]);
    const float wz = fmaf((float)gz + 0.5f, g.voxel, g.origin[2]);
    unsigned in = 0u;
#pragma unroll
    for (int j = 0; j < VEC; j++)
        if (lut_pixel<ORD>(v, fmaf((float)(gx + j) + 0.5f, g.voxel, g.origin[0]), wy, wz, &cam[j], &pix[j])) in |= 1u << j;
#pragma unroll
    for (int j = 0; j < VEC; j++) packed[j] = in >> j & 1u ? __ldg(depth + pix[j]) : 0u;
    return in;
}

/* VEC values at p, 16 bytes at once where VEC is 4 (u16: 8). */
template <int VEC>
__device__ __forceinline__ void load_quad(const float* p, float* o) {
    if (VEC == 4) {
        const float4 a = *(const float4*)p;
        o[0] = a.x;
        o[1 % VEC] = a.y;
        o[2 % VEC] = a.z;
        o[3 % VEC] = a.w;
    } else {
        o[0] = *p;
    }
}
template <int VEC>
__device__ __forceinline__ void store_quad(float* p, const float* o) {
    if (VEC == 4) *(float4*)p = make_float4(o[0], o[1 % VEC], o[2 % VEC], o[3 % VEC]);
    else *p = o[0];
}
template <int VEC>
__device__ __forceinline__ void load_quad(const uint16_t* p, uint32_t* o) {
    if (VEC == 4) {
        const ushort4 a = *(const ushort4*)p;
        o[0] = a.x;
        o[1 % VEC] = a.y;
        o[2 % VEC] = a.z;
        o[3 % VEC] = a.w;
    } else {
        o[0] = *p;
    }
}
template <int VEC>
__device__ __forceinline__ void store_quad(uint16_t* p, const uint32_t* o) {
    if (VEC == 4)
        *(ushort4*)p = make_ushort4((uint16_t)o[0], (uint16_t)o[1 % VEC], (uint16_t)o[2 % VEC], (uint16_t)o[3 % VEC]);
    else
        *p = (uint16_t)o[0];
}

/* Out-of-place integration of one view: (tsdf_in, weight_in) -> (tsdf_out, weight_out), every
 * voxel written (in place when the pointers are equal).  Same culling and arithmetic as
 * k_integrate.  Bound by the volume's reads and writes: a thread per four voxels, in brick-major
 * order (a culled brick is a copy), 256^3 voxels with f32 weights 73 us (3.7 TB/s); a voxel per thread
 * with 64-bit index divisions and general divisions was bound by issue, 142 us. */
template <int VEC, bool Q8, bool ORD>
__global__ void __launch_bounds__(256) k_integrate_depth(const L3dTsdfGrid g, const L3dTsdfView v,
                                                         const int32_t* __restrict__ coords,
                                                         const uint8_t* __restrict__ mask,
                                                         const uint32_t* __restrict__ depth,
                                                         const float* __restrict__ depthf,
                                                         const float* __restrict__ prior,
                                                         const float4* __restrict__ normals,
                                                         const float* tsdf_in, const void* weight_in,
                                                         float* tsdf_out, void* weight_out,
                                                         long long quads) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= quads) return;
    int gx, gy, gz;
    long long idx, brick;
    if (!quad_coords<VEC>(g, coords, q, &gx, &gy, &gz, &idx, &brick)) return;
    float t[VEC], wf[VEC];
    uint32_t wq[VEC];
    load_quad<VEC>(tsdf_in + idx, t);
    if (Q8) load_quad<VEC>((const uint16_t*)weight_in + idx, wq);
    else load_quad<VEC>((const float*)weight_in + idx, wf);
    if (mask[brick]) {
        float3 cam[VEC];
        PixelIndex<ORD> pix[VEC];
        uint32_t packed[VEC];
        const unsigned in = quad_pixels<VEC, ORD>(g, v, depth, gx, gy, gz, cam, pix, packed);
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            float obs, w, dobs, dw;
            if (!(in >> j & 1u) || !observe_diff<ORD>(g, v, depthf, v.has_prior ? prior : nullptr, normals, cam[j],
                                                      packed[j], &pix[j], &obs, &w, &dobs, &dw))
                continue;
            if (Q8) apply_q8(t[j], wq[j], obs, w, g.max_q);
            else apply_f32(t[j], wf[j], obs, w, g.max_weight);
        }
    }
    store_quad<VEC>(tsdf_out + idx, t);
    if (Q8) store_quad<VEC>((uint16_t*)weight_out + idx, wq);
    else store_quad<VEC>((float*)weight_out + idx, wf);
}

/* Adjoint of k_integrate_depth.  Per voxel, with the state (T0, W0) before the update and the
 * observation o(d) with weight w(d):
 *   T1 = (T0 W0 + o w) / (W0 + w),  W1 = min(W0 + w, max)
 *   dT1/dT0 = W0 / (W0 + w),  dT1/dW0 = (T0 - T1) / (W0 + w)
 *   dT1/dd  = (w do/dd + (o - T1) dw/dd) / (W0 + w),  dW1/dd = dw/dd, dW1/dW0 = 1 (below max)
 * gT, gW are the loss gradients with respect to T1 and W1 (gW may be NULL).  The depth gradient
 * is added into grad_depth with atomics (many voxels see one pixel); grad_tsdf_in and
 * grad_weight_in (either may be NULL) are written for every voxel.  Q8.8 weights are integers:
 * dw/dd and the weight gradients are zero there.  Laid out like the forward kernel; the state is read
 * only where the view updates it (256^3 voxels 77 us, before 153 us). */
template <int VEC, bool Q8, bool ORD>
__global__ void __launch_bounds__(256) k_integrate_depth_grad(
        const L3dTsdfGrid g, const L3dTsdfView v, const int32_t* __restrict__ coords,
        const uint8_t* __restrict__ mask, const uint32_t* __restrict__ depth,
        const float* __restrict__ depthf, const float* __restrict__ prior, const float4* __restrict__ normals,
        const float* __restrict__ tsdf_in, const void* __restrict__ weight_in,
        const float* __restrict__ gT, const float* __restrict__ gW, float* __restrict__ grad_depth,
        float* __restrict__ grad_tsdf_in, float* __restrict__ grad_weight_in, long long quads) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= quads) return;
    int gx, gy, gz;
    long long idx, brick;
    if (!quad_coords<VEC>(g, coords, q, &gx, &gy, &gz, &idx, &brick)) return;
    float gt[VEC], gw[VEC];
    load_quad<VEC>(gT + idx, gt);
#pragma unroll
    for (int j = 0; j < VEC; j++) gw[j] = 0.0f;
    if (!Q8 && gW) load_quad<VEC>(gW + idx, gw);
    if (mask[brick]) {
        float3 cam[VEC];
        PixelIndex<ORD> pix[VEC];
        uint32_t packed[VEC];
        const unsigned in = quad_pixels<VEC, ORD>(g, v, depth, gx, gy, gz, cam, pix, packed);
#pragma unroll
        for (int j = 0; j < VEC; j++) {
            float obs, w, dobs, dw;
            if (!(in >> j & 1u) || !observe_diff<ORD>(g, v, depthf, v.has_prior ? prior : nullptr, normals, cam[j],
                                                      packed[j], &pix[j], &obs, &w, &dobs, &dw))
                continue;
            float w0, wu = w;
            if (Q8) {
                const uint32_t wi = (uint32_t)rintf(w * 256.0f);
                if (wi == 0u) continue;
                w0 = (float)((const uint16_t*)weight_in)[idx + j] * 0.00390625f;
                wu = (float)wi * 0.00390625f;
                dw = 0.0f;
            } else {
                w0 = ((const float*)weight_in)[idx + j];
            }
            const float t0 = tsdf_in[idx + j];
            const float den = w0 + wu;
            const float t1 = fmaf(t0, w0, obs * wu) / den;
            const float below = (!Q8 && (w0 + wu < g.max_weight)) ? 1.0f : 0.0f;
            const float gtj = gt[j], gwj = gw[j];
            gt[j] = gtj * (w0 / den);
            gw[j] = fmaf(gtj, (t0 - t1) / den, gwj * below);
            if (pix[j] >= 0 && grad_depth) {
                const float gd = gtj * (fmaf(wu, dobs, (obs - t1) * dw) / den) + gwj * below * dw;
                if (gd != 0.0f) atomicAdd(grad_depth + pix[j], gd);
            }
        }
    }
    if (grad_tsdf_in) store_quad<VEC>(grad_tsdf_in + idx, gt);
    if (grad_weight_in) {
        if (Q8) {
#pragma unroll
            for (int j = 0; j < VEC; j++) gw[j] = 0.0f;
        }
        store_quad<VEC>(grad_weight_in + idx, gw);
    }
}

/* tsdf 1 and weight 0, 16 bytes per store (both buffers start on 16 bytes); bound by the writes: 805 MB
 * of 512^3 voxels with Q8.8 weights 128 us, a voxel per thread 273 us. */
__global__ void __launch_bounds__(256) k_fill(float* tsdf, void* weight, long long voxels, int q8) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x, n = (long long)gridDim.x * blockDim.x;
    for (long long k = i; k < voxels / 4; k += n) ((float4*)tsdf)[k] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    const long long words = voxels * (q8 ? 2 : 4) / 16;
    for (long long k = i; k < words; k += n) ((uint4*)weight)[k] = make_uint4(0u, 0u, 0u, 0u);
    /* what does not fill 16 bytes */
    if (i < voxels % 4) tsdf[voxels - 1 - i] = 1.0f;
    if (q8 && i < voxels % 8) ((uint16_t*)weight)[voxels - 1 - i] = 0;
    if (!q8 && i < voxels % 4) ((float*)weight)[voxels - 1 - i] = 0.0f;
}

}  // namespace

bool l3d_tsdf_ordinary(const L3dTsdfGrid& g, const L3dTsdfView* views, int n) {
    if (!(g.mu >= 0x1p-60f && g.mu <= 0x1p60f)) return false;
    /* the largest magnitude of a voxel centre's coordinate on each axis (brick coordinates are int32) */
    double reach[3];
    for (int i = 0; i < 3; i++)
        reach[i] = std::fabs(g.origin_d[i]) + (g.dense ? (double)g.dims[i] + 8.0 : 0x1p35) * g.voxel_d;
    for (int k = 0; k < n; k++) {
        const L3dTsdfView& v = views[k];
        if (v.W > 1 << 22 || v.H > 1 << 22 || (long long)v.W * v.H >= 1ll << 31) return false;
        for (int r = 0; r < 3; r++) {
            double bound = std::fabs((double)v.t[r]);
            for (int i = 0; i < 3; i++) bound += std::fabs((double)v.R[r * 3 + i]) * reach[i];
            if (!(bound < 0x1p50)) return false;
        }
    }
    return true;
}

namespace {

inline bool vec4_ok(const L3dTsdfGrid& g) { return !g.dense || (g.dims[0] % 4 == 0); }

/* Threads of the integration kernels (brick-major order, see quad_coords). */
inline long long quad_count(const L3dTsdfGrid& g, int vec) {
    return g.bricks * (512 / vec);
}

}  // namespace

cudaError_t l3d_launch_tsdf_visible(const L3dTsdfGrid& g, const L3dTsdfView* views_dev, int n_views,
                                    const int32_t* coords, uint8_t* mask, cudaStream_t stream) {
    long long n = g.bricks * mask_stride(n_views);
    if (n == 0 || n_views == 0) return cudaSuccess;
    k_visible<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(g, views_dev, n_views, coords, mask);
    return cudaGetLastError();
}

long long l3d_depth_tile_count(int W, int H) {
    return (long long)((W + L3D_DEPTH_TILE - 1) / L3D_DEPTH_TILE) * ((H + L3D_DEPTH_TILE - 1) / L3D_DEPTH_TILE);
}

cudaError_t l3d_launch_depth_tiles(const L3dTsdfView* views_dev, int n_views,
                                   const uint32_t* const* depth_ptrs_dev, const float* priors,
                                   float* tiles, long long max_tiles, cudaStream_t stream) {
    if (n_views <= 0 || max_tiles <= 0) return cudaSuccess;
    dim3 grid((unsigned)((max_tiles * 8 + 127) / 128), (unsigned)n_views);
    k_depth_tiles<<<grid, 128, 0, stream>>>(views_dev, n_views, depth_ptrs_dev, priors, tiles, max_tiles);
    return cudaGetLastError();
}

long long l3d_tsdf_super_pairs(const L3dTsdfGrid& g, int n_views) {
    if (!g.dense) return 0;
    const long long n = (long long)super_count(g, 0) * super_count(g, 1) * super_count(g, 2) * n_views;
    return n < (1ll << 32) ? n : 0;  /* a pair is one u32 */
}

int l3d_tsdf_visible_launches(const L3dTsdfGrid& g, int n_views) { return l3d_tsdf_super_pairs(g, n_views) > 0 ? 2 : 1; }

cudaError_t l3d_launch_tsdf_visible_depth(const L3dTsdfGrid& g, const L3dTsdfView* views_dev, int n_views,
                                          const int32_t* coords, const float* tiles, uint32_t* pairs,
                                          uint8_t* mask, cudaStream_t stream) {
    long long n = g.bricks * mask_stride(n_views);
    if (n == 0 || n_views == 0) return cudaSuccess;
    const long long np = l3d_tsdf_super_pairs(g, n_views);
    if (np == 0) {
        k_visible_depth<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(g, views_dev, n_views, coords, tiles, mask);
        return cudaGetLastError();
    }
    cudaError_t e;
    if ((e = cudaMemsetAsync(pairs, 0, sizeof(uint32_t), stream)) != cudaSuccess ||
        (e = cudaMemsetAsync(mask, 0, (size_t)n, stream)) != cudaSuccess)
        return e;
    k_super_pairs<<<(unsigned)((np * 8 + 255) / 256), 256, 0, stream>>>(g, views_dev, n_views, tiles, pairs);
    const unsigned blocks = (unsigned)std::min<long long>(148 * 8, (np * 64 + 255) / 256);
    k_visible_pairs<<<blocks, 256, 0, stream>>>(g, views_dev, n_views, tiles, pairs, mask);
    return cudaGetLastError();
}

cudaError_t l3d_launch_tsdf_view(const L3dTsdfGrid& g, const L3dTsdfView& v, const int32_t* coords,
                                 uint8_t* mask, const uint32_t* depth, const float* prior,
                                 const float4* normals, float* tiles, int32_t* list, float* tsdf,
                                 void* weight, int q8, cudaStream_t stream) {
    if (g.bricks == 0) return cudaSuccess;
    if (tiles && list && normals && l3d_tsdf_ordinary(g, &v, 1)) {
        /* kept bricks only: tiles, the listing cull, a grid-stride sweep of the listed bricks */
        const long long nt = l3d_depth_tile_count(v.W, v.H);
        L3dTsdfView vt = v;
        vt.tile_off = 0;
        k_depth_tiles_one<<<(unsigned)((nt * 8 + 127) / 128), 128, 0, stream>>>(vt, depth, prior, tiles, list);
        cudaError_t e;
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if (g.bricks <= LANES_BRICKS)
            k_visible_one_list<true><<<(unsigned)((g.bricks * 8 + 127) / 128), 128, 0, stream>>>(g, vt, coords, tiles, list);
        else
            k_visible_one_list<false><<<(unsigned)((g.bricks + 127) / 128), 128, 0, stream>>>(g, vt, coords, tiles, list);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const unsigned blocks = (unsigned)std::min<long long>(148 * 8, (g.bricks * 128 + 255) / 256);
        if (vec4_ok(g)) {
            if (q8) k_integrate_list<4, true><<<blocks, 256, 0, stream>>>(g, v, coords, list, depth, prior, normals, tsdf, weight);
            else k_integrate_list<4, false><<<blocks, 256, 0, stream>>>(g, v, coords, list, depth, prior, normals, tsdf, weight);
        } else {
            if (q8) k_integrate_list<1, true><<<blocks, 256, 0, stream>>>(g, v, coords, list, depth, prior, normals, tsdf, weight);
            else k_integrate_list<1, false><<<blocks, 256, 0, stream>>>(g, v, coords, list, depth, prior, normals, tsdf, weight);
        }
        return cudaGetLastError();
    }
    k_visible_one<<<(unsigned)((g.bricks + 255) / 256), 256, 0, stream>>>(g, v, coords, mask);
    const int vec = vec4_ok(g) ? 4 : 1;
    long long quads = quad_count(g, vec);
    if (quads == 0) return cudaSuccess;
    unsigned blocks = (unsigned)((quads + 255) / 256);
#define L3D_INTEGRATE(V, Q, L) \
    k_integrate<V, Q, L><<<blocks, 256, 0, stream>>>(g, v, coords, mask, depth, prior, normals, tsdf, weight, quads)
    if (normals) {
        if (vec == 4) {
            if (q8) L3D_INTEGRATE(4, true, true);
            else L3D_INTEGRATE(4, false, true);
        } else {
            if (q8) L3D_INTEGRATE(1, true, true);
            else L3D_INTEGRATE(1, false, true);
        }
    } else {
        if (vec == 4) {
            if (q8) L3D_INTEGRATE(4, true, false);
            else L3D_INTEGRATE(4, false, false);
        } else {
            if (q8) L3D_INTEGRATE(1, true, false);
            else L3D_INTEGRATE(1, false, false);
        }
    }
#undef L3D_INTEGRATE
    return cudaGetLastError();
}

cudaError_t l3d_launch_tsdf_count(const L3dTsdfGrid& g, const L3dTsdfView* views_dev, int n_views,
                                  const int32_t* coords, const uint8_t* mask,
                                  const uint32_t* const* depth_ptrs_dev, const float* priors,
                                  const float4* normals, unsigned long long* counts,
                                  cudaStream_t stream) {
    const int vec = vec4_ok(g) ? 4 : 1;
    long long quads = quad_count(g, vec);
    if (quads == 0 || n_views == 0) return cudaSuccess;
    unsigned blocks = (unsigned)((quads + 255) / 256);
    if (vec == 4)
        k_count_updates<4><<<blocks, 256, 0, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, quads, counts);
    else
        k_count_updates<1><<<blocks, 256, 0, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, quads, counts);
    return cudaGetLastError();
}

cudaError_t l3d_launch_normal_table(float4* normals, cudaStream_t stream) {
    k_normal_table<<<16, 256, 0, stream>>>(normals);
    return cudaGetLastError();
}

long long l3d_tsdf_sweep_units(const L3dTsdfGrid& g, long long* layer_units, long long* layer_voxels) {
    const int vec = vec4_ok(g) ? 4 : 1;
    if (g.dense) {
        if (layer_units) *layer_units = (long long)g.nb[0] * g.nb[1] * (512 / vec);
        if (layer_voxels) *layer_voxels = 8ll * g.dims[0] * g.dims[1];
    } else {
        if (layer_units) *layer_units = 512 / vec;
        if (layer_voxels) *layer_voxels = 512;
    }
    return quad_count(g, vec);
}

cudaError_t l3d_launch_tsdf_many_range(const L3dTsdfGrid& g, const L3dTsdfView* views_dev,
                                       int n_views, const int32_t* coords, const uint8_t* mask,
                                       const uint32_t* const* depth_ptrs_dev, const float* priors,
                                       const float4* normals, float* tsdf, void* weight, int q8,
                                       long long q_begin, long long q_end, cudaStream_t stream) {
    const int vec = vec4_ok(g) ? 4 : 1;
    q_end = q_end < quad_count(g, vec) ? q_end : quad_count(g, vec);
    if (q_end <= q_begin || n_views == 0) return cudaSuccess;
    unsigned blocks = (unsigned)((q_end - q_begin + 255) / 256);
    if (vec == 4) {
        if (q8) k_integrate_many<4, true><<<blocks, 256, 0, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, q_begin, q_end);
        else k_integrate_many<4, false><<<blocks, 256, 0, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, q_begin, q_end);
    } else {
        if (q8) k_integrate_many<1, true><<<blocks, 256, 0, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, q_begin, q_end);
        else k_integrate_many<1, false><<<blocks, 256, 0, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, q_begin, q_end);
    }
    return cudaGetLastError();
}

cudaError_t l3d_launch_tsdf_brick_list(const L3dTsdfGrid& g, int n_views, const uint8_t* mask,
                                      uint32_t* flags, uint32_t* prefix, int32_t* list,
                                      uint32_t* scratch, cudaStream_t stream) {
    if (g.bricks == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((g.bricks + 1 + 255) / 256);
    k_brick_any<<<blocks, 256, 0, stream>>>(mask, mask_stride(n_views), g.bricks, flags);
    cudaError_t e = l3d_scan_exclusive(flags, prefix, g.bricks + 1, scratch, nullptr, stream);
    if (e != cudaSuccess) return e;
    k_brick_list_fill<<<blocks, 256, 0, stream>>>(flags, prefix, g.bricks, list);
    return cudaGetLastError();
}

cudaError_t l3d_launch_tsdf_many_list(const L3dTsdfGrid& g, const L3dTsdfView* views_dev,
                                      int n_views, const int32_t* coords, const uint8_t* mask,
                                      const uint32_t* const* depth_ptrs_dev, const float* priors,
                                      const float4* normals, float* tsdf, void* weight, int q8,
                                      const uint32_t* prefix, const int32_t* list, uint32_t* next,
                                      bool ordinary, long long q_begin, long long q_end, cudaStream_t stream) {
    const int vec = vec4_ok(g) ? 4 : 1;
    const long long per = 512 / vec;
    q_end = q_end < quad_count(g, vec) ? q_end : quad_count(g, vec);
    if (q_end <= q_begin || n_views == 0) return cudaSuccess;
    const long long b0 = q_begin / per, b1 = (q_end + per - 1) / per;
    /* four resident blocks per SM, passes handed out as warps ask */
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 148;
    const unsigned blocks = (unsigned)(4 * sms);
    const size_t smem = (size_t)n_views * sizeof(L3dTsdfView);
    /* more than ~200 views, or numbers out of the ordinary: the sweep of every quad, views from global
     * memory */
    if (smem > 48 * 1024 || !ordinary)
        return l3d_launch_tsdf_many_range(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors,
                                          normals, tsdf, weight, q8, q_begin, q_end, stream);
    /* where even all bricks kept are no more than the fixed rounds, no warp asks */
    if ((b1 - b0) * (per / 32) > (long long)blocks * 8 * kFixedRounds) {
        const cudaError_t e = cudaMemsetAsync(next, 0, sizeof(uint32_t), stream);
        if (e != cudaSuccess) return e;
    }
    if (vec == 4) {
        if (q8) k_integrate_many_list<4, true><<<blocks, 256, smem, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, prefix, list, next, b0, b1);
        else k_integrate_many_list<4, false><<<blocks, 256, smem, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, prefix, list, next, b0, b1);
    } else {
        if (q8) k_integrate_many_list<1, true><<<blocks, 256, smem, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, prefix, list, next, b0, b1);
        else k_integrate_many_list<1, false><<<blocks, 256, smem, stream>>>(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors, normals, tsdf, weight, prefix, list, next, b0, b1);
    }
    return cudaGetLastError();
}

cudaError_t l3d_launch_tsdf_many(const L3dTsdfGrid& g, const L3dTsdfView* views_dev, int n_views,
                                 const int32_t* coords, const uint8_t* mask,
                                 const uint32_t* const* depth_ptrs_dev, const float* priors,
                                 const float4* normals, float* tsdf, void* weight, int q8,
                                 cudaStream_t stream) {
    return l3d_launch_tsdf_many_range(g, views_dev, n_views, coords, mask, depth_ptrs_dev, priors,
                                      normals, tsdf, weight, q8, 0, l3d_tsdf_sweep_units(g, nullptr, nullptr),
                                      stream);
}

namespace {
template <int VEC, bool Q8, bool ORD>
cudaError_t launch_depth(const L3dTsdfGrid& g, const L3dTsdfView& v, const int32_t* coords, const uint8_t* mask,
                         const uint32_t* depth, const float* depthf, const float* prior, const float4* normals,
                         const float* tsdf_in, const void* weight_in, float* tsdf_out, void* weight_out,
                         const float* grad_tsdf_out, const float* grad_weight_out, float* grad_depth,
                         float* grad_tsdf_in, float* grad_weight_in, cudaStream_t stream) {
    const long long quads = quad_count(g, VEC);
    const unsigned blocks = (unsigned)((quads + 255) / 256);
    if (grad_tsdf_out)
        k_integrate_depth_grad<VEC, Q8, ORD><<<blocks, 256, 0, stream>>>(g, v, coords, mask, depth, depthf, prior, normals, tsdf_in, weight_in, grad_tsdf_out, grad_weight_out, grad_depth, grad_tsdf_in, grad_weight_in, quads);
    else
        k_integrate_depth<VEC, Q8, ORD><<<blocks, 256, 0, stream>>>(g, v, coords, mask, depth, depthf, prior, normals, tsdf_in, weight_in, tsdf_out, weight_out, quads);
    return cudaGetLastError();
}
}  // namespace

cudaError_t l3d_launch_tsdf_depth(const L3dTsdfGrid& g, const L3dTsdfView& v, const int32_t* coords,
                                  uint8_t* mask, const uint32_t* depth, const float* depthf,
                                  const float* prior, const float4* normals, const float* tsdf_in,
                                  const void* weight_in, float* tsdf_out, void* weight_out,
                                  const float* grad_tsdf_out, const float* grad_weight_out,
                                  float* grad_depth, float* grad_tsdf_in, float* grad_weight_in, int q8,
                                  cudaStream_t stream) {
    if (g.bricks == 0) return cudaSuccess;
    k_visible_one<<<(unsigned)((g.bricks + 255) / 256), 256, 0, stream>>>(g, v, coords, mask);
    /* four voxels at once where the grid's rows and the caller's tensors allow 16-byte accesses */
    size_t low = 0;
    for (const void* p : {(const void*)tsdf_in, weight_in, (const void*)tsdf_out, (const void*)weight_out,
                          (const void*)grad_tsdf_out, (const void*)grad_weight_out, (const void*)grad_tsdf_in,
                          (const void*)grad_weight_in})
        low |= (size_t)p & 15;
    const bool vec = vec4_ok(g) && low == 0, ord = l3d_tsdf_ordinary(g, &v, 1);
#define L3D_DEPTH(V, Q, O) \
    launch_depth<V, Q, O>(g, v, coords, mask, depth, depthf, prior, normals, tsdf_in, weight_in, tsdf_out, weight_out, grad_tsdf_out, grad_weight_out, grad_depth, grad_tsdf_in, grad_weight_in, stream)
    if (!ord) return q8 ? L3D_DEPTH(1, true, false) : L3D_DEPTH(1, false, false);
    if (vec) return q8 ? L3D_DEPTH(4, true, true) : L3D_DEPTH(4, false, true);
    return q8 ? L3D_DEPTH(1, true, true) : L3D_DEPTH(1, false, true);
#undef L3D_DEPTH
}

cudaError_t l3d_launch_tsdf_fill(float* tsdf, void* weight, long long voxels, int q8,
                                 cudaStream_t stream) {
    if (voxels == 0) return cudaSuccess;
    k_fill<<<(unsigned)std::min<long long>((voxels / 4 + 255) / 256 + 1, 148 * 16), 256, 0, stream>>>(tsdf, weight, voxels, q8);
    return cudaGetLastError();
}

/*
 * Surface extraction on the device: naive surface nets on the TSDF volume in place, area-weighted
 * vertex normals, removal of small connected components, and the brick grid that allocates a
 * volume around a point cloud.
 *
 * frontend/src/app/vision/fusion/surface-nets.ts:47-174 walks the pool brick by brick, voxel by
 * voxel, appending one vertex per cell whose eight corners are observed and change sign, then
 * one quad per sign-changing voxel edge.  The reference's append order is kept: vertex k of the
 * output is the k-th flagged cell in (brick, local voxel) order, and the triangles come in (brick,
 * voxel, axis) order.  Which cells are flagged and which edges carry a quad depends on two bits per
 * voxel alone (observed, negative), so the volume is read once, into those bits (1/24 of it), and the
 * rest works on them, a warp per brick and a byte per row of eight voxels: flags, counts per brick,
 * one prefix sum over the bricks, and then only the bricks that hold surface emit vertices and
 * triangles, one lane per vertex or quad.  A volume of 384^3 (12 views, 39 thousand vertices) took 1.66 ms
 * of kernels when each pass ran a thread per cell over five arrays of 4 bytes per cell, and takes
 * 0.19 ms, a third of it the one read of the volume.
 *
 * Positions are computed in FP64 and rounded to f32 like the reference's number[] ->
 * Float32Array; the quad diagonal is chosen on the FP64 positions.
 *
 * Normals (mesh.ts:9-31): the reference adds each face's FP64 cross product into f32 vertex
 * sums in face order.  Each vertex gathers its faces (a CSR of vertex -> faces, each list sorted
 * by face index) and sums them in that order, so the f32 sums round exactly as the reference's.
 *
 * Components (mesh.ts:37-87): union-find over the faces' edges (l3d_labels.h: one root is hooked onto the
 * other with a compare-and-swap, paths are shortened on the way); the kept faces keep their order and
 * vertices are renumbered in order of first use, as the reference's union-find pass does.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "l3d_internal.h"
#include "l3d_labels.h"

namespace {

constexpr int BV = 512;

struct Cell {
    int x, y, z;
};

__device__ __forceinline__ void brick_origin(const L3dSdfView& v, long long b, int* x0, int* y0, int* z0) {
    if (v.dense) {
        *x0 = (int)(b % v.dims[0]) * 8;
        *y0 = (int)((b / v.dims[0]) % v.dims[1]) * 8;
        *z0 = (int)(b / ((long long)v.dims[0] * v.dims[1])) * 8;
    } else {
        *x0 = v.coords[b * 4] * 8;
        *y0 = v.coords[b * 4 + 1] * 8;
        *z0 = v.coords[b * 4 + 2] * 8;
    }
}

/* Storage index of voxel (x, y, z), -1 when it does not exist (the reference's slot()). */
__device__ __forceinline__ long long storage_of(const L3dSdfView& v, int x, int y, int z) {
    if (x < 0 || y < 0 || z < 0 || x >= v.vdims[0] || y >= v.vdims[1] || z >= v.vdims[2]) return -1;
    if (v.dense) return ((long long)z * v.vdims[1] + y) * v.vdims[0] + x;
    const int brick = v.lookup[((long long)(z >> 3) * v.dims[1] + (y >> 3)) * v.dims[0] + (x >> 3)];
    if (brick < 0) return -1;
    return (long long)brick * BV + (x & 7) + ((y & 7) << 3) + ((z & 7) << 6);
}

__constant__ int kCorner[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {1, 1, 0},
                                  {0, 0, 1}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}};
__constant__ int kEdge[12][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3},
                                 {4, 6}, {5, 7}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

constexpr int kWarps = 8;  /* warps (bricks) per block of the surface kernels */

/* The brick that holds the voxels at brick coordinates (bx, by, bz), -1 when there is none. */
__device__ __forceinline__ int brick_at(const L3dSdfView& v, int bx, int by, int bz) {
    if (bx < 0 || by < 0 || bz < 0 || bx >= v.dims[0] || by >= v.dims[1] || bz >= v.dims[2]) return -1;
    const long long i = ((long long)bz * v.dims[1] + by) * v.dims[0] + bx;
    return v.dense ? (int)i : v.lookup[i];
}

/* Eight voxels of a row as bits (bit x): `n` of them exist.  ALIGNED: the row is complete and its start
 * aligned for 16-byte loads of f32 and 8-byte loads of u16. */
template <bool ALIGNED, bool Q8>
__device__ __forceinline__ uint32_t observed_row(const L3dSdfView& v, long long at, int n) {
    uint32_t bits = 0u;
    if (ALIGNED && Q8) {
        const ushort4* p = (const ushort4*)((const uint16_t*)v.weight + at);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const ushort4 w = __ldg(p + k);
            const uint16_t q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (!((float)q[j] * 0.00390625f < v.min_weight_f)) bits |= 1u << (4 * k + j);
        }
    } else if (ALIGNED) {
        const float4* p = (const float4*)((const float*)v.weight + at);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const float4 w = __ldg(p + k);
            const float q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (!(q[j] < v.min_weight_f)) bits |= 1u << (4 * k + j);
        }
    } else {
        for (int x = 0; x < n; x++) {
            const float w = Q8 ? (float)((const uint16_t*)v.weight)[at + x] * 0.00390625f
                               : ((const float*)v.weight)[at + x];
            if (!(w < v.min_weight_f)) bits |= 1u << x;
        }
    }
    return bits;
}
template <bool ALIGNED>
__device__ __forceinline__ uint32_t negative_row(const L3dSdfView& v, long long at, int n) {
    uint32_t bits = 0u;
    if (ALIGNED) {
        const float4* p = (const float4*)(v.tsdf + at);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const float4 t = __ldg(p + k);
            bits |= ((t.x < 0.0f ? 1u : 0u) | (t.y < 0.0f ? 2u : 0u) | (t.z < 0.0f ? 4u : 0u) |
                     (t.w < 0.0f ? 8u : 0u)) << (4 * k);
        }
    } else {
        for (int x = 0; x < n; x++)
            if (v.tsdf[at + x] < 0.0f) bits |= 1u << x;
    }
    return bits;
}

/* The bits of a brick's voxels, by storage brick: a warp per brick, two rows per lane (`lane` and
 * `lane` + 32).  The tsdf is read only where the brick has an observed voxel.  Bound by the loads: two
 * rows in 16-byte pieces per lane (384^3, Q8.8 weights: a load and a ballot per voxel took 168 us). */
template <bool ALIGNED, bool Q8>
__global__ void __launch_bounds__(32 * kWarps) k_sn_bits(const L3dSdfView v, long long bricks, uint32_t* obs,
                                                         uint32_t* neg) {
    const long long b = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (b >= bricks) return;
    const int lane = threadIdx.x & 31;
    long long at[2];
    int n[2] = {8, 8};
    if (v.dense) {
        int x0, y0, z0;
        brick_origin(v, b, &x0, &y0, &z0);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int y = y0 + (lane & 7), z = z0 + (lane >> 3) + 4 * k;
            at[k] = ((long long)z * v.vdims[1] + y) * v.vdims[0] + x0;
            n[k] = y < v.vdims[1] && z < v.vdims[2] ? min(8, v.vdims[0] - x0) : 0;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 2; k++) at[k] = b * BV + (lane + 32 * k) * 8;
    }
    uint32_t o[2] = {0u, 0u}, m[2] = {0u, 0u};
#pragma unroll
    for (int k = 0; k < 2; k++)
        if (n[k]) o[k] = observed_row<ALIGNED, Q8>(v, at[k], n[k]);
    if (__any_sync(0xffffffffu, (o[0] | o[1]) != 0u)) {
#pragma unroll
        for (int k = 0; k < 2; k++)
            if (n[k]) m[k] = negative_row<ALIGNED>(v, at[k], n[k]) & o[k];
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        ((uint8_t*)obs)[b * 64 + lane + 32 * k] = (uint8_t)o[k];
        ((uint8_t*)neg)[b * 64 + lane + 32 * k] = (uint8_t)m[k];
    }
}

__device__ __forceinline__ uint32_t row_of(const uint32_t* words, int brick, int y, int z) {
    return brick < 0 ? 0u : ((const uint8_t*)words)[(size_t)brick * 64 + y + 8 * z];
}

/* Nine rows on each of y and z and nine bits along x of one kind of bits, from the brick and its
 * neighbours: row (y, z), 0 <= y, z <= 8, at [y + 9 z], bit x of 0..8.  nb[dx + 2 dy + 4 dz] are the brick
 * and the next ones along each axis. */
__device__ __forceinline__ void rows_ahead(const uint32_t* words, const int* nb, uint16_t* rows) {
    for (int i = threadIdx.x & 31; i < 81; i += 32) {
        const int y = i % 9, z = i / 9, k = (y == 8 ? 2 : 0) + (z == 8 ? 4 : 0);
        rows[i] = (uint16_t)(row_of(words, nb[k], y & 7, z & 7) | (row_of(words, nb[k + 1], y & 7, z & 7) & 1u) << 8);
    }
}
/* The same looking back: row (y, z), -1 <= y, z <= 7, at [(y + 1) + 9 (z + 1)], bit x + 1 for -1 <= x <= 7;
 * nb are the brick and the previous ones along each axis. */
__device__ __forceinline__ void rows_behind(const uint32_t* words, const int* nb, uint16_t* rows) {
    for (int i = threadIdx.x & 31; i < 81; i += 32) {
        const int y = i % 9 - 1, z = i / 9 - 1, k = (y < 0 ? 2 : 0) + (z < 0 ? 4 : 0);
        rows[i] = (uint16_t)(row_of(words, nb[k], y & 7, z & 7) << 1 | row_of(words, nb[k + 1], y & 7, z & 7) >> 7);
    }
}

/* nb[8] of the warp's brick: the bricks at +-1 along each axis (step +1 or -1). */
__device__ __forceinline__ void neighbours(const L3dSdfView& v, long long b, int step, int* nb) {
    const int lane = threadIdx.x & 31;
    if (lane < 8) {
        int x0, y0, z0;
        brick_origin(v, b, &x0, &y0, &z0);
        nb[lane] = brick_at(v, (x0 >> 3) + step * (lane & 1), (y0 >> 3) + step * ((lane >> 1) & 1),
                            (z0 >> 3) + step * (lane >> 2));
    }
    __syncwarp();
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

/* Exclusive sums over a brick's 64 rows, two per lane (rows lane and lane + 32); returns the total. */
__device__ __forceinline__ uint32_t row_prefix(uint32_t a, uint32_t c, uint32_t* pa, uint32_t* pc) {
    const int lane = threadIdx.x & 31;
    uint32_t ia = a, ic = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t ta = __shfl_up_sync(0xffffffffu, ia, off), tc = __shfl_up_sync(0xffffffffu, ic, off);
        if (lane >= off) {
            ia += ta;
            ic += tc;
        }
    }
    const uint32_t first = __shfl_sync(0xffffffffu, ia, 31);
    *pa = ia - a;
    *pc = first + ic - c;
    return first + __shfl_sync(0xffffffffu, ic, 31);
}

/* sampleCell (surface-nets.ts:79-88) of every cell of a brick: its eight corners observed and not all of
 * one sign. */
__global__ void __launch_bounds__(32 * kWarps) k_sn_flags(const L3dSdfView v, long long bricks, const L3dSurfaceBits t) {
    __shared__ int nbs[kWarps][8];
    __shared__ uint16_t obs[kWarps][81], neg[kWarps][81];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long b = (long long)blockIdx.x * kWarps + warp;
    if (b >= bricks) return;
    int* nb = nbs[warp];
    neighbours(v, b, 1, nb);
    uint8_t* out = (uint8_t*)t.flag + (size_t)b * 64;
    const uint32_t own = nb[0] >= 0 && lane < 16 ? t.obs[(size_t)nb[0] * 16 + lane] : 0u;
    if (!__any_sync(0xffffffffu, own != 0u)) {  /* a cell's first corner is its own voxel */
        out[lane] = 0;
        out[lane + 32] = 0;
        if (lane == 0) t.count[b] = 0ull;
        return;
    }
    rows_ahead(t.obs, nb, obs[warp]);
    rows_ahead(t.neg, nb, neg[warp]);
    __syncwarp();
    uint32_t f[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int r = lane + 32 * k, i = (r & 7) + 9 * (r >> 3);
        const uint16_t *o = obs[warp] + i, *n = neg[warp] + i;
        const uint32_t seen = o[0] & o[1] & o[9] & o[10];
        const uint32_t some = n[0] | n[1] | n[9] | n[10], all = n[0] & n[1] & n[9] & n[10];
        f[k] = seen & seen >> 1 & (some | some >> 1) & ~(all & all >> 1) & 255u;
        out[r] = (uint8_t)f[k];
    }
    uint32_t pa, pc;
    const uint32_t total = row_prefix(__popc(f[0]), __popc(f[1]), &pa, &pc);
    if (total) {
        t.rank[b * 64 + lane] = (uint16_t)pa;
        t.rank[b * 64 + lane + 32] = (uint16_t)pc;
    }
    if (lane == 0) t.count[b] = total;
}

/* The voxel edges of a row that carry a quad (surface-nets.ts:120-165), a bit per voxel and axis: the edge's
 * ends have different signs and its four cells are flagged (a flagged cell's corners are observed, so
 * the ends are).  i: the row's place in `flag` (rows_behind) and `neg` (rows_ahead). */
__device__ __forceinline__ void row_edges(const uint16_t* flag, const uint16_t* neg, int row, uint32_t* e) {
    const int y = row & 7, z = row >> 3;
    const uint16_t* f = flag + (y + 1) + 9 * (z + 1);
    const uint16_t* n = neg + y + 9 * z;
    const uint32_t f00 = f[0], fy = f[-1], fz = f[-9], fyz = f[-10], n0 = n[0];
    e[0] = (n0 ^ n0 >> 1) & (f00 & fy & fz & fyz) >> 1 & 255u;
    e[1] = (n0 ^ n[1]) & (f00 & fz) >> 1 & f00 & fz & 255u;
    e[2] = (n0 ^ n[9]) & (f00 & fy) >> 1 & f00 & fy & 255u;
}

/* Quads per brick, added to count[] (high half). */
__global__ void __launch_bounds__(32 * kWarps) k_sn_quads(const L3dSdfView v, long long bricks, const L3dSurfaceBits t) {
    __shared__ int nbs[kWarps][8];
    __shared__ uint16_t flag[kWarps][81], neg[kWarps][81];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long b = (long long)blockIdx.x * kWarps + warp;
    if (b >= bricks) return;
    const unsigned long long vertices = t.count[b];
    if (!vertices) return;  /* a quad's last cell is its own voxel's */
    neighbours(v, b, -1, nbs[warp]);
    rows_behind(t.flag, nbs[warp], flag[warp]);
    __syncwarp();
    neighbours(v, b, 1, nbs[warp]);
    rows_ahead(t.neg, nbs[warp], neg[warp]);
    __syncwarp();
    uint32_t n = 0;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        uint32_t e[3];
        row_edges(flag[warp], neg[warp], lane + 32 * k, e);
        n += __popc(e[0]) + __popc(e[1]) + __popc(e[2]);
    }
    n = warp_sum(n);
    if (lane == 0) t.count[b] = vertices | (unsigned long long)n << 32;
}

/* The last of 64 rows with prefix[row] <= i, prefix ascending from 0. */
__device__ __forceinline__ int row_holding(const uint16_t* prefix, uint32_t i) {
    int row = 0;
#pragma unroll
    for (int step = 32; step > 0; step >>= 1)
        if (prefix[row + step] <= i) row += step;
    return row;
}

/* Pass 1 (surface-nets.ts:90-118): the vertex of each flagged cell, a lane per vertex; degree[] is
 * cleared for pass 2. */
__global__ void __launch_bounds__(32 * kWarps) k_sn_vertex(const L3dSdfView v, long long bricks, const L3dSurfaceBits t,
                                                           double* pos_d, float* pos_f, uint32_t* degree) {
    __shared__ uint16_t prefix[kWarps][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long b = (long long)blockIdx.x * kWarps + warp;
    if (b >= bricks) return;
    const uint32_t count = (uint32_t)t.count[b], base = (uint32_t)t.base[b];
    if (!count) return;
    prefix[warp][lane] = t.rank[b * 64 + lane];
    prefix[warp][lane + 32] = t.rank[b * 64 + lane + 32];
    __syncwarp();
    int x0, y0, z0;
    brick_origin(v, b, &x0, &y0, &z0);
    for (uint32_t i = lane; i < count; i += 32) {
        const int row = row_holding(prefix[warp], i);
        uint32_t bits = ((const uint8_t*)t.flag)[(size_t)b * 64 + row];
        for (uint32_t k = i - prefix[warp][row]; k > 0; k--) bits &= bits - 1u;
        const int x = x0 + __ffs(bits) - 1, y = y0 + (row & 7), z = z0 + (row >> 3);
        double values[8];
#pragma unroll
        for (int c = 0; c < 8; c++)
            values[c] = (double)v.tsdf[storage_of(v, x + kCorner[c][0], y + kCorner[c][1], z + kCorner[c][2])];
        double sx = 0.0, sy = 0.0, sz = 0.0;
        int n = 0;
#pragma unroll
        for (int e = 0; e < 12; e++) {
            const int a = kEdge[e][0], d = kEdge[e][1];
            const double va = values[a], vc = values[d];
            if ((va < 0.0) == (vc < 0.0)) continue;
            const double s = va / (va - vc);
            sx += kCorner[a][0] + (kCorner[d][0] - kCorner[a][0]) * s;
            sy += kCorner[a][1] + (kCorner[d][1] - kCorner[a][1]) * s;
            sz += kCorner[a][2] + (kCorner[d][2] - kCorner[a][2]) * s;
            n++;
        }
        const double p[3] = {v.origin[0] + (x + 0.5 + sx / n) * v.voxel,
                             v.origin[1] + (y + 0.5 + sy / n) * v.voxel,
                             v.origin[2] + (z + 0.5 + sz / n) * v.voxel};
        const size_t k = (size_t)base + i;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            pos_d[k * 3 + q] = p[q];
            pos_f[k * 3 + q] = (float)p[q];
        }
        degree[k] = 0u;
    }
}

__device__ __forceinline__ double dist2(const double* p, uint32_t a, uint32_t b) {
    const double dx = p[(size_t)a * 3] - p[(size_t)b * 3];
    const double dy = p[(size_t)a * 3 + 1] - p[(size_t)b * 3 + 1];
    const double dz = p[(size_t)a * 3 + 2] - p[(size_t)b * 3 + 2];
    return dx * dx + dy * dy + dz * dz;
}

/* One triangle: its indices, its normal in FP64 (the cross product of mesh.ts:15-21, from the f32
 * positions) and a count at its vertices. */
__device__ __forceinline__ void put_face(uint32_t i0, uint32_t i1, uint32_t i2, const float* p, uint32_t* idx,
                                         double* fn, uint32_t* degree) {
    const size_t a = (size_t)i0 * 3, b = (size_t)i1 * 3, c = (size_t)i2 * 3;
    const double e1[3] = {(double)p[b] - p[a], (double)p[b + 1] - p[a + 1], (double)p[b + 2] - p[a + 2]};
    const double e2[3] = {(double)p[c] - p[a], (double)p[c + 1] - p[a + 1], (double)p[c + 2] - p[a + 2]};
    fn[0] = e1[1] * e2[2] - e1[2] * e2[1];
    fn[1] = e1[2] * e2[0] - e1[0] * e2[2];
    fn[2] = e1[0] * e2[1] - e1[1] * e2[0];
    idx[0] = i0;
    idx[1] = i1;
    idx[2] = i2;
    atomicAdd(degree + i0, 1u);
    atomicAdd(degree + i1, 1u);
    atomicAdd(degree + i2, 1u);
}

/* Pass 2 (surface-nets.ts:120-165): the two triangles of each quad, a lane per quad. */
__global__ void __launch_bounds__(32 * kWarps) k_sn_emit(const L3dSdfView v, long long bricks, const L3dSurfaceBits t,
                                                         const double* pos_d, const float* pos_f, uint32_t* indices,
                                                         double* fn, uint32_t* degree) {
    __shared__ int back[kWarps][8], ahead[kWarps][8];
    __shared__ uint16_t flag[kWarps][81], neg[kWarps][81], prefix[kWarps][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long b = (long long)blockIdx.x * kWarps + warp;
    if (b >= bricks) return;
    const uint32_t count = (uint32_t)(t.count[b] >> 32), base = (uint32_t)(t.base[b] >> 32);
    if (!count) return;
    const int* nb = back[warp];
    neighbours(v, b, -1, back[warp]);
    neighbours(v, b, 1, ahead[warp]);
    rows_behind(t.flag, back[warp], flag[warp]);
    rows_ahead(t.neg, ahead[warp], neg[warp]);
    __syncwarp();
    uint32_t e[3], n[2], pa, pc;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        row_edges(flag[warp], neg[warp], lane + 32 * k, e);
        n[k] = __popc(e[0]) + __popc(e[1]) + __popc(e[2]);
    }
    row_prefix(n[0], n[1], &pa, &pc);
    prefix[warp][lane] = (uint16_t)pa;
    prefix[warp][lane + 32] = (uint16_t)pc;
    __syncwarp();
    /* the vertex of the cell at (x, y, z), -1 <= x, y, z <= 7: its brick's base, the flagged cells in the
     * rows before and in the row before it */
    auto vertex = [&](int x, int y, int z) {
        const int brick = nb[(x < 0 ? 1 : 0) + (y < 0 ? 2 : 0) + (z < 0 ? 4 : 0)];
        const size_t row = (size_t)brick * 64 + (y & 7) + 8 * (z & 7);
        const uint32_t bits = ((const uint8_t*)t.flag)[row];
        return (uint32_t)t.base[brick] + t.rank[row] + __popc(bits & ((1u << (x & 7)) - 1u));
    };
    for (uint32_t i = lane; i < count; i += 32) {
        const int row = row_holding(prefix[warp], i), y = row & 7, z = row >> 3;
        row_edges(flag[warp], neg[warp], row, e);
        int x = 0, a = 0;
        for (uint32_t k = i - prefix[warp][row];;) {  /* the k-th edge of the row, by voxel, then axis */
            if (e[a] >> x & 1u) {
                if (k == 0) break;
                k--;
            }
            if (++a == 3) {
                a = 0;
                x++;
            }
        }
        /* axes b = a + 1 and d = a + 2 (mod 3) step to the edge's other cells */
        const int ux = a == 2, uy = a == 0, uz = a == 1, wx = a == 1, wy = a == 2, wz = a == 0;
        const uint32_t q0 = vertex(x - ux - wx, y - uy - wy, z - uz - wz), q2 = vertex(x, y, z);
        const uint32_t qw = vertex(x - wx, y - wy, z - wz), qu = vertex(x - ux, y - uy, z - uz);
        const bool inside = (neg[warp][y + 9 * z] >> x & 1u) != 0u;
        const uint32_t q1 = inside ? qw : qu, q3 = inside ? qu : qw;
        const size_t o = ((size_t)base + i) * 6;
        const bool along = dist2(pos_d, q0, q2) <= dist2(pos_d, q1, q3);
        put_face(q0, q1, along ? q2 : q3, pos_f, indices + o, fn + o, degree);
        put_face(along ? q0 : q1, q2, q3, pos_f, indices + o + 3, fn + o + 3, degree);
    }
}

/* ---- normals ---- */

/* Each vertex's faces, in any order; end[] starts at the lists' beginnings and ends at their ends. */
__global__ void k_face_lists(const uint32_t* idx, long long faces, uint32_t* end, uint32_t* lists) {
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= faces) return;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t v = idx[f * 3 + k];
        lists[atomicAdd(end + v, 1u)] = (uint32_t)f;
    }
}

/* computeNormals: each vertex sums its faces in face order into f32, then normalises. */
__global__ void k_vertex_normals(long long vertices, const uint32_t* end, const uint32_t* degree,
                                 uint32_t* lists, const double* fn, float* nrm) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= vertices) return;
    const uint32_t n = degree[v];
    uint32_t* l = lists + (end[v] - n);
    for (uint32_t i = 1; i < n; i++) {  /* insertion sort: a handful of faces per vertex */
        const uint32_t key = l[i];
        uint32_t j = i;
        while (j > 0 && l[j - 1] > key) {
            l[j] = l[j - 1];
            j--;
        }
        l[j] = key;
    }
    float s[3] = {0.0f, 0.0f, 0.0f};
    for (uint32_t i = 0; i < n; i++) {
        const double* f = fn + (size_t)l[i] * 3;
#pragma unroll
        for (int k = 0; k < 3; k++) s[k] = (float)((double)s[k] + f[k]);
    }
    double length = sqrt((double)s[0] * s[0] + (double)s[1] * s[1] + (double)s[2] * s[2]);
    if (!(length != 0.0)) length = 1.0;
#pragma unroll
    for (int k = 0; k < 3; k++) nrm[v * 3 + k] = (float)((double)s[k] / length);
}

/* ---- components ---- */

__global__ void k_cc_init(long long vertices, uint32_t* label) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < vertices) label[v] = (uint32_t)v;
}

/* Labels in global memory.  Other threads change them meanwhile, so every access is one relaxed operation
 * that the compiler neither repeats nor merges with another. */
struct GlobalLabels {
    uint32_t* label;
    __device__ __forceinline__ uint32_t load(uint32_t v) const {
        uint32_t l;
        asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(l) : "l"(label + v) : "memory");
        return l;
    }
    __device__ __forceinline__ void store(uint32_t v, uint32_t l) const {
        asm volatile("st.relaxed.gpu.u32 [%0], %1;" : : "l"(label + v), "r"(l) : "memory");
    }
    __device__ __forceinline__ bool swap(uint32_t v, uint32_t from, uint32_t to) const {
        return atomicCAS(label + v, from, to) == from;
    }
};

__global__ void k_cc_unite(const uint32_t* idx, long long faces, uint32_t* label, int* err) {
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= faces) return;
    const uint32_t a = idx[f * 3], b = idx[f * 3 + 1], c = idx[f * 3 + 2];
    GlobalLabels m = {label};
    l3d_label_unite(m, a, b, err);
    l3d_label_unite(m, b, c, err);
}

__global__ void k_cc_flatten(long long vertices, uint32_t* label, int* err) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    GlobalLabels m = {label};
    if (v < vertices) l3d_label_flatten(m, (uint32_t)v, err);
}

/* Faces per component; the lanes of a warp that share one add once. */
__global__ void k_cc_count(const uint32_t* idx, long long faces, const uint32_t* label,
                           uint32_t* comp_faces) {
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = f < faces;
    const unsigned active = __ballot_sync(0xffffffffu, in);
    if (!in) return;
    const uint32_t l = label[idx[f * 3]];
    const unsigned same = __match_any_sync(active, l);
    if ((int)(threadIdx.x & 31u) == __ffs(same) - 1) atomicAdd(comp_faces + l, (uint32_t)__popc(same));
}

/* first[v] = first corner position (3f + k) of a kept face that uses v */
__global__ void k_cc_keep(const uint32_t* idx, long long faces, const uint32_t* label,
                          const uint32_t* comp_faces, double limit, uint32_t* first) {
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= faces || !((double)comp_faces[label[idx[f * 3]]] >= limit)) return;
#pragma unroll
    for (int q = 0; q < 3; q++) atomicMin(first + idx[f * 3 + q], (uint32_t)(f * 3 + q));
}

/* kept faces and first uses, packed for one prefix sum */
__global__ void k_cc_pack(const uint32_t* idx, long long faces, const uint32_t* label,
                          const uint32_t* comp_faces, double limit, const uint32_t* first,
                          unsigned long long* pack) {
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= faces) return;
    const bool kept = (double)comp_faces[label[idx[f * 3]]] >= limit;
    unsigned long long n = 0;
#pragma unroll
    for (int q = 0; q < 3; q++) n += first[idx[f * 3 + q]] == (uint32_t)(f * 3 + q) ? 1u : 0u;
    pack[f] = (kept ? 1ull : 0ull) | n << 32;
}

__global__ void k_cc_emit(const uint32_t* idx, long long faces, const unsigned long long* pack,
                          const unsigned long long* base, const uint32_t* first, const float* pos,
                          const float* nrm, uint32_t* out_idx, float* out_pos, float* out_nrm) {
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= faces || !((uint32_t)pack[f])) return;
    const size_t o = (size_t)(uint32_t)base[f] * 3;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const uint32_t v = idx[f * 3 + q], at = first[v];
        /* v's number: the first uses before its own */
        const uint32_t face = at / 3;
        uint32_t r = (uint32_t)(base[face] >> 32);
        for (uint32_t k = face * 3; k < at; k++) r += first[idx[k]] == k ? 1u : 0u;
        out_idx[o + q] = r;
        if (at == (uint32_t)(f * 3 + q)) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                out_pos[(size_t)r * 3 + k] = pos[(size_t)v * 3 + k];
                out_nrm[(size_t)r * 3 + k] = nrm[(size_t)v * 3 + k];
            }
        }
    }
}

/* ---- brick grid (tsdf-volume.ts:36-64) ---- */

__global__ void k_grid_mark(const float* pts, long long n, L3dBrickGrid g, double radius, uint8_t* marks) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double side = g.voxel * 8.0;
    int lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double p = (double)pts[i * 3 + k];
        lo[k] = (int)fmax(0.0, floor((p - radius - g.origin[k]) / side));
        hi[k] = (int)fmin((double)(g.dims[k] - 1), floor((p + radius - g.origin[k]) / side));
    }
    for (int bz = lo[2]; bz <= hi[2]; bz++)
        for (int by = lo[1]; by <= hi[1]; by++)
            for (int bx = lo[0]; bx <= hi[0]; bx++)
                marks[((long long)bz * g.dims[1] + by) * g.dims[0] + bx] = 1;
}

__global__ void k_grid_widen(const uint8_t* marks, long long cells, uint32_t* flags) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < cells) flags[i] = marks[i] ? 1u : 0u;
}

__global__ void k_grid_build(const uint32_t* flags, const uint32_t* base, long long cells, L3dBrickGrid g,
                             int32_t* lookup, int32_t* coords) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    if (!flags[i]) {
        lookup[i] = -1;
        return;
    }
    const uint32_t b = base[i];
    lookup[i] = (int32_t)b;
    if (coords) {
        coords[(size_t)b * 4] = (int32_t)(i % g.dims[0]);
        coords[(size_t)b * 4 + 1] = (int32_t)((i / g.dims[0]) % g.dims[1]);
        coords[(size_t)b * 4 + 2] = (int32_t)(i / ((long long)g.dims[0] * g.dims[1]));
        coords[(size_t)b * 4 + 3] = 0;
    }
}

inline unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }

}  // namespace

cudaError_t l3d_launch_sn_bits(const L3dSdfView& v, long long bricks, const L3dSurfaceBits& t, cudaStream_t s) {
    if (!bricks) return cudaSuccess;
    const unsigned n = (unsigned)((bricks + kWarps - 1) / kWarps);
    /* rows of a dense grid are whole and aligned where X is a multiple of 8 */
    const bool aligned = (!v.dense || v.vdims[0] % 8 == 0) && ((size_t)v.tsdf & 15) == 0 && ((size_t)v.weight & 15) == 0;
    if (aligned && v.q8) k_sn_bits<true, true><<<n, 32 * kWarps, 0, s>>>(v, bricks, t.obs, t.neg);
    else if (aligned) k_sn_bits<true, false><<<n, 32 * kWarps, 0, s>>>(v, bricks, t.obs, t.neg);
    else if (v.q8) k_sn_bits<false, true><<<n, 32 * kWarps, 0, s>>>(v, bricks, t.obs, t.neg);
    else k_sn_bits<false, false><<<n, 32 * kWarps, 0, s>>>(v, bricks, t.obs, t.neg);
    k_sn_flags<<<n, 32 * kWarps, 0, s>>>(v, bricks, t);
    k_sn_quads<<<n, 32 * kWarps, 0, s>>>(v, bricks, t);
    return cudaGetLastError();
}
cudaError_t l3d_launch_sn_emit(const L3dSdfView& v, long long bricks, const L3dSurfaceBits& t, double* pos_d,
                               float* pos_f, uint32_t* indices, double* fn, uint32_t* degree, cudaStream_t s) {
    if (!bricks) return cudaSuccess;
    const unsigned n = (unsigned)((bricks + kWarps - 1) / kWarps);
    k_sn_vertex<<<n, 32 * kWarps, 0, s>>>(v, bricks, t, pos_d, pos_f, degree);
    k_sn_emit<<<n, 32 * kWarps, 0, s>>>(v, bricks, t, pos_d, pos_f, indices, fn, degree);
    return cudaGetLastError();
}
cudaError_t l3d_launch_vertex_normals(const uint32_t* idx, long long faces, long long vertices, uint32_t* start,
                                      const uint32_t* degree, uint32_t* lists, const double* fn, float* nrm,
                                      cudaStream_t s) {
    if (faces) k_face_lists<<<blocks_for(faces), 256, 0, s>>>(idx, faces, start, lists);
    if (vertices) k_vertex_normals<<<blocks_for(vertices), 256, 0, s>>>(vertices, start, degree, lists, fn, nrm);
    return cudaGetLastError();
}
cudaError_t l3d_launch_cc_labels(const uint32_t* idx, long long faces, long long vertices, uint32_t* label,
                                 int* err, cudaStream_t s) {
    if (!vertices) return cudaSuccess;
    k_cc_init<<<blocks_for(vertices), 256, 0, s>>>(vertices, label);
    if (faces) k_cc_unite<<<blocks_for(faces), 256, 0, s>>>(idx, faces, label, err);
    k_cc_flatten<<<blocks_for(vertices), 256, 0, s>>>(vertices, label, err);
    return cudaGetLastError();
}
cudaError_t l3d_launch_cc_keep(const uint32_t* idx, long long faces, const uint32_t* label,
                               uint32_t* comp_faces, double limit, uint32_t* first,
                               unsigned long long* pack, cudaStream_t s) {
    if (!faces) return cudaSuccess;
    k_cc_count<<<blocks_for(faces), 256, 0, s>>>(idx, faces, label, comp_faces);
    k_cc_keep<<<blocks_for(faces), 256, 0, s>>>(idx, faces, label, comp_faces, limit, first);
    k_cc_pack<<<blocks_for(faces), 256, 0, s>>>(idx, faces, label, comp_faces, limit, first, pack);
    return cudaGetLastError();
}
cudaError_t l3d_launch_cc_emit(const uint32_t* idx, long long faces, const unsigned long long* pack,
                               const unsigned long long* base, const uint32_t* first,
                               const float* pos, const float* nrm, uint32_t* out_idx, float* out_pos,
                               float* out_nrm, cudaStream_t s) {
    if (faces)
        k_cc_emit<<<blocks_for(faces), 256, 0, s>>>(idx, faces, pack, base, first, pos, nrm, out_idx, out_pos,
                                                    out_nrm);
    return cudaGetLastError();
}
cudaError_t l3d_launch_grid_mark(const float* pts, long long n, const L3dBrickGrid& g, double radius,
                                 uint8_t* marks, cudaStream_t s) {
    if (n) k_grid_mark<<<blocks_for(n), 256, 0, s>>>(pts, n, g, radius, marks);
    return cudaGetLastError();
}
cudaError_t l3d_launch_grid_widen(const uint8_t* marks, long long cells, uint32_t* flags, cudaStream_t s) {
    if (cells) k_grid_widen<<<blocks_for(cells), 256, 0, s>>>(marks, cells, flags);
    return cudaGetLastError();
}
cudaError_t l3d_launch_grid_build(const uint32_t* flags, const uint32_t* base, long long cells,
                                  const L3dBrickGrid& g, int32_t* lookup, int32_t* coords, cudaStream_t s) {
    if (cells) k_grid_build<<<blocks_for(cells), 256, 0, s>>>(flags, base, cells, g, lookup, coords);
    return cudaGetLastError();
}

/*
 * Where a warped matching window lies in a source image, decided from its four corners.
 *
 * The exact evaluators (plain and exact forms, gradients) take a window as lost when any of its
 * samples has q.z <= 1e-6 or lies outside [0, W-1] x [0, H-1], each position computed in FP32 as
 * q.xy / q.z, q = H (x, y, 1).  The window's image is the convex hull of its corners' images, so
 * corners that are inside by more than the rounding of a position stand for every sample, and a
 * corner that is outside by as much (the corners are samples) loses the window.  The bound: each
 * component of q carries two roundings of a sum whose magnitudes are mx, my, mz, the quotient two
 * more, so a position is off by at most (3 mx + wmax mz) 2^-23 / q.z; sixteen such units are
 * allowed.  What is neither (a window that grazes a border, and anything that has left the ordinary
 * numbers, NaN included: every comparison with it fails) tests its samples one by one.
 */
#ifndef L3D_WINDOW_CUH
#define L3D_WINDOW_CUH

#include <cuda_runtime.h>

#include "l3d_ieee.h"

enum L3dPlace { L3D_INSIDE, L3D_OUTSIDE, L3D_GRAZES };

/* h: the homography, row-major; (px, py) >= 0 the window's centre, e its half size; wmax, hmax the
 * source's last texel coordinates.  Inside, q.z lies in [1e-6, 2^121] and every bilinear footprint
 * within the image. */
__device__ __forceinline__ L3dPlace l3d_window_place(const float* h, float px, float py, float e, float wmax,
                                                     float hmax) {
    float zmin = 3.0e38f, zmax = -3.0e38f, umin = 3.0e38f, umax = -3.0e38f, vmin = 3.0e38f, vmax = -3.0e38f;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const float x = px + ((c & 1) ? e : -e);
        const float y = py + ((c & 2) ? e : -e);
        const float qz = fmaf(h[6], x, fmaf(h[7], y, h[8]));
        const float iz = l3d_rcp_approx(qz);
        const float u = fmaf(h[0], x, fmaf(h[1], y, h[2])) * iz;
        const float v = fmaf(h[3], x, fmaf(h[4], y, h[5])) * iz;
        zmin = fminf(zmin, qz);
        zmax = fmaxf(zmax, qz);
        umin = fminf(umin, u);
        umax = fmaxf(umax, u);
        vmin = fminf(vmin, v);
        vmax = fmaxf(vmax, v);
    }
    const float ax = px + e, ay = py + e;
    const float mx = fmaf(fabsf(h[0]), ax, fmaf(fabsf(h[1]), ay, fabsf(h[2])));
    const float my = fmaf(fabsf(h[3]), ax, fmaf(fabsf(h[4]), ay, fabsf(h[5])));
    const float mz = fmaf(fabsf(h[6]), ax, fmaf(fabsf(h[7]), ay, fabsf(h[8])));
    const float unit = 0x1p-20f * l3d_rcp_approx(zmin);
    const float su = unit * fmaf(wmax, mz, mx), sv = unit * fmaf(hmax, mz, my);
    /* strictly below the last texel, whose footprint has no right or lower neighbour: su is 0 where a row of
     * H is, and the window of such an H lies on one texel of an image one pixel wide */
    if (zmin > fmaf(0x1p-20f, mz, 1e-6f) && zmax < 0x1p120f && umin >= su && vmin >= sv && umax < wmax - su &&
        vmax < hmax - sv)
        return L3D_INSIDE;
    if (zmin <= 1e-6f || umin < -su || vmin < -sv || umax > wmax + su || vmax > hmax + sv) return L3D_OUTSIDE;
    return L3D_GRAZES;
}

#endif

/* l3d_window_place (csrc/l3d_window.cuh) on the host, beside the per-sample tests it stands for.  The
 * hardware reciprocal (within one ulp) is the rounded one moved by `off` ulps. */
#include <math.h>
#include <stdint.h>
#include <string.h>

#define __device__
#define __forceinline__ inline
#define L3D_IEEE_H
static int off;
static float l3d_rcp_approx(float x) {
    float y = 1.0f / x;
    if (fabsf(y) < 1.17549435e-38f) return copysignf(0.0f, y);  /* flushed */
    for (int i = 0; i < off; i++) y = nextafterf(y, INFINITY);
    for (int i = 0; i > off; i--) y = nextafterf(y, -INFINITY);
    return y;
}
#include "l3d_window.cuh"

/* counts[0]: windows found inside, [1] outside, [2] neither; [3] inside ones with a sample that is lost or
 * whose bilinear footprint leaves the image; [4] outside ones without a lost sample. */
extern "C" void window_places(int n, const float* h9, const float* pxy, int side, int dilation, int W, int H, int ulps,
                              int* counts) {
    off = ulps;
    const int half = (side - 1) * dilation / 2;
    const float wmax = (float)(W - 1), hmax = (float)(H - 1);
    for (int i = 0; i < n; i++) {
        const float* h = h9 + i * 9;
        const float px = pxy[2 * i], py = pxy[2 * i + 1];
        const L3dPlace place = l3d_window_place(h, px, py, (float)half, wmax, hmax);
        bool lost = false, leaves = false;
        for (int k = 0; k < side * side; k++) {
            const float x = px + (float)(k % side * dilation - half), y = py + (float)(k / side * dilation - half);
            const float qz = fmaf(h[6], x, fmaf(h[7], y, h[8]));
            const float iz = 1.0f / qz;
            const float u = fmaf(h[0], x, fmaf(h[1], y, h[2])) * iz, v = fmaf(h[3], x, fmaf(h[4], y, h[5])) * iz;
            if (!(qz > 1e-6f && u >= 0.0f && v >= 0.0f && u <= wmax && v <= hmax)) lost = true;
            else if (floorf(u) + 1.0f > wmax || floorf(v) + 1.0f > hmax) leaves = true;
        }
        counts[place == L3D_INSIDE ? 0 : place == L3D_OUTSIDE ? 1 : 2]++;
        if (place == L3D_INSIDE && (lost || leaves)) counts[3]++;
        if (place == L3D_OUTSIDE && !lost) counts[4]++;
    }
}

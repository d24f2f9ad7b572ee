/*
 * Image preparation on the device, in front of the stereo stage: RGBA -> gray with area
 * downsampling, RGB thumbnails, gray downsampling, and upsampling of the phone's depth grid into a
 * stereo prior.
 *
 *   frontend/src/app/vision/image/gray-image.ts:12-46    rgbaToGray
 *   frontend/src/app/vision/image/gray-image.ts:49-82    downsampleRgb
 *   frontend/src/app/vision/image/gray-image.ts:166-187  downsampleGray
 *   frontend/src/app/vision/image/gray-image.ts:193-239  resampleArea, coverage
 *   frontend/src/app/vision/mvs/depth-maps.ts:9-42       upsampleDepth
 * Arithmetic follows the reference: integer luma sums, FP64 weights and sums, f32 intermediate rows,
 * round-half-up (floor, plus one when the fraction is at least 1/2) and truncating byte stores.
 * The area filter's per-pixel coverage tables (first source pixel and weights) are computed on
 * the host in FP64 like the reference's coverage().
 *
 * A frame's kernels are a few microseconds each, so launches and the latency of a thread's loads bound
 * them, not memory: blocks of source pixels are shared by lanes, means are integer divisions (exact, see
 * k_blocks), and the area filter is one launch where its footprint is small.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "l3d_internal.h"

namespace {

__device__ __forceinline__ double js_round(double x) {
    const double f = floor(x);
    return (x - f >= 0.5) ? f + 1.0 : f;
}

__device__ __forceinline__ uint8_t to_u8(double v) {
    const double t = trunc(v);
    return (uint8_t)(t - 256.0 * floor(t / 256.0));
}

__device__ __forceinline__ void block_bounds(int t, double s, int* a, int* b) {
    *a = (int)floor(t * s);
    *b = max(*a + 1, (int)floor((t + 1) * s));
}

/* Pixel i of an RGBA image: one load where the image starts on a 4-byte boundary. */
template <bool WORDS>
__device__ __forceinline__ uint32_t rgba_at(const uint8_t* __restrict__ src, long long i) {
    if (WORDS) return __ldg((const uint32_t*)src + i);
    const uint8_t* p = src + i * 4;
    return p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16;
}
/* 77 r + 150 g + 29 b */
__device__ __forceinline__ uint32_t luma256(uint32_t px) { return __dp4a(px, 0x001d964du, 0u); }

enum BlockKind { BLOCK_LUMA, BLOCK_RGB, BLOCK_GRAY };

/* Means over blocks of source pixels: rgbaToGray's and downsampleGray's integer-ratio paths
 * (gray-image.ts:26-45, 170-186) and downsampleRgb (gray-image.ts:49-82).  The reference divides an
 * integer sum by an integer count in FP64 and rounds half up (gray) or truncates (RGB); counts are below
 * 2^31 and quotients at most 255, so the quotient's rounding (2^-45) never reaches the next half or
 * integer (2^-40 away at least, or equal), and the integer division gives the same byte.
 * 2^shift lanes share a block's columns: a lane alone walks a 32 x 32 block in 1024 steps (1280 x 960 to
 * 40 x 30: 141 us, with 32 lanes 19; to a 160 x 120 thumbnail 11.4 -> 7.2 us, with FP64 sums and
 * divisions before).  ALONE: one lane per block, its loads at constant steps (8000 x 6000 gray to 1000 x 750:
 * 16.4 us, 22.6 with the step in a register; not for RGB, whose 2 x 2 blocks it slows).  WIDE: sums beyond 32 bits. */
template <int KIND, bool WORDS, bool WIDE, bool ALONE>
__global__ void __launch_bounds__(256) k_blocks(const uint8_t* __restrict__ src, int W, int H, int tw, int th, double sx,
                                                double sy, int shift, uint8_t* __restrict__ out) {
    using sum_t = typename std::conditional<WIDE, unsigned long long, uint32_t>::type;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long pixels = (long long)tw * th;
    const int lanes = ALONE ? 1 : 1 << shift, lane = ALONE ? 0 : (int)t & (lanes - 1);
    const long long o = ALONE ? t : t >> shift;
    const int i = (int)(o < pixels ? o : pixels - 1); /* every lane takes part in the sums */
    const int y = i / tw, x = i - y * tw;
    int x0, x1, y0, y1;
    block_bounds(x, sx, &x0, &x1);
    block_bounds(y, sy, &y0, &y1);
    sum_t a = 0, b = 0, c = 0;
    for (int yy = y0; yy < y1; yy++) {
        const long long row = (long long)yy * W;
#pragma unroll (KIND == BLOCK_GRAY && ALONE ? 4 : 2)
        for (int xx = x0 + lane; xx < x1; xx += lanes) {
            if (KIND == BLOCK_GRAY) {
                a += src[row + xx];
            } else {
                const uint32_t px = rgba_at<WORDS>(src, row + xx);
                if (KIND == BLOCK_LUMA) {
                    a += luma256(px);
                } else {
                    a += px & 255u;
                    b += px >> 8 & 255u;
                    c += px >> 16 & 255u;
                }
            }
        }
    }
    for (int k = lanes >> 1; k > 0; k >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, k);
        if (KIND == BLOCK_RGB) {
            b += __shfl_xor_sync(0xffffffffu, b, k);
            c += __shfl_xor_sync(0xffffffffu, c, k);
        }
    }
    if (lane != 0 || o >= pixels) return;
    const sum_t n = (sum_t)(y1 - y0) * (sum_t)(x1 - x0);
    if (KIND == BLOCK_RGB) {
        out[o * 3] = (uint8_t)(a / n);
        out[o * 3 + 1] = (uint8_t)(b / n);
        out[o * 3 + 2] = (uint8_t)(c / n);
    } else {
        const sum_t d = KIND == BLOCK_LUMA ? n * 256u : n;
        out[o] = (uint8_t)((2 * a + d) / (2 * d));
    }
}

/* source pixel as the area filter reads it: u8 gray, or the f32 luma of an RGBA pixel
 * (rgbaToGray's Float32Array store, gray-image.ts:20-23; exact: 16 bits over 256) computed on the fly */
template <bool RGBA, bool WORDS>
__device__ __forceinline__ float area_src(const uint8_t* __restrict__ src, long long i) {
    if (!RGBA) return (float)src[i];
    return (float)luma256(rgba_at<WORDS>(src, i)) * 0.00390625f;
}

/* resampleArea pass 1 (gray-image.ts:203-212): rows of the source -> f32 temp (tw per row).
 * cover: per target column, first source pixel and `k` weights (stride `kmax`). */
template <bool RGBA, bool WORDS>
__global__ void k_area_rows(const uint8_t* __restrict__ src, int W, int H, int tw, const L3dAreaCover cols,
                            float* __restrict__ temp) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)tw * H) return;
    const int x = (int)(i % tw);
    const long long y = i / tw;
    const long long row = y * W + cols.first[x];
    const double* w = cols.weights + (size_t)x * cols.kmax;
    double sum = 0.0;
    for (int k = 0; k < cols.count[x]; k++) sum += w[k] * (double)area_src<RGBA, WORDS>(src, row + k);
    temp[i] = (float)sum;
}

/* resampleArea pass 2 (gray-image.ts:213-220): columns of the temp -> bytes */
__global__ void k_area_cols(const float* __restrict__ temp, int tw, int th, const L3dAreaCover rows,
                            uint8_t* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tw * th) return;
    const int x = i % tw, y = i / tw;
    const double* w = rows.weights + (size_t)y * rows.kmax;
    double sum = 0.0;
    for (int k = 0; k < rows.count[y]; k++) sum += w[k] * (double)temp[(size_t)(rows.first[y] + k) * tw + x];
    out[i] = to_u8(fmin(255.0, js_round(sum)));
}

/* Both passes at once, a thread per output pixel: the row sums of its source rows, in the passes'
 * operations and order.  A row on a boundary is summed for both outputs, which costs less than the second
 * launch and the intermediate's allocation and trip while footprints are at most AREA_TAPS each way
 * (1280 x 960 to 600 x 450: 12.8 us in two passes, 9.8 in one, back to back 16.0 and 8.4; 7 taps: 10.4 and
 * 9.7).  Larger footprints, whose targets are small images, keep the two passes: a thread walks the whole
 * footprint alone (9 taps: 13.3 and 14.0; 22 taps: 21 and 54).  So do large targets, where the row sums made
 * twice cost more than the launch: from 1.5 million pixels of gray bytes (1280 x 960 to 1440 x 1080: 21.9 us in
 * one pass, 20.5 in two; 4000 x 3000 to 4500 x 3375: 179 and 135) and 2 million of RGBA, whose row sums also
 * take the luma twice (1600 x 1200: 24.7 either way; 4500 x 3375: 164 and 150).  SMALL: at most four taps. */
constexpr int AREA_TAPS = 8;
constexpr long long AREA_GRAY = 1500000, AREA_RGBA = 2000000;
template <bool RGBA, bool WORDS, bool SMALL>
__global__ void __launch_bounds__(256) k_area(const uint8_t* __restrict__ src, int W, int tw, int th,
                                              const L3dAreaCover cols, const L3dAreaCover rows,
                                              uint8_t* __restrict__ out) {
    const unsigned across = (unsigned)(tw + 31) / 32;
    const int x = (int)(blockIdx.x % across) * 32 + threadIdx.x, y = (int)(blockIdx.x / across) * 8 + threadIdx.y;
    if (x >= tw || y >= th) return;
    const int fx = cols.first[x], nx = cols.count[x], fy = rows.first[y], ny = rows.count[y];
    const double* wx = cols.weights + (size_t)x * cols.kmax;
    const double* wy = rows.weights + (size_t)y * rows.kmax;
    const long long at = (long long)fy * W + fx;
    double sum = 0.0;
    if (SMALL) {
        /* the whole footprint's loads in flight before the first sum */
        double c[4], r[4];
        float v[4][4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            c[j] = j < nx ? wx[j] : 0.0;
            r[j] = j < ny ? wy[j] : 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++) v[j][k] = j < ny && k < nx ? area_src<RGBA, WORDS>(src, at + (long long)j * W + k) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j >= ny) break;
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < nx) s += c[k] * (double)v[j][k];
            sum += r[j] * (double)(float)s;
        }
    } else {
        for (int j = 0; j < ny; j++) {
            double s = 0.0;
            for (int k = 0; k < nx; k++) s += wx[k] * (double)area_src<RGBA, WORDS>(src, at + (long long)j * W + k);
            sum += wy[j] * (double)(float)s;
        }
    }
    out[(size_t)y * tw + x] = to_u8(fmin(255.0, js_round(sum)));
}

/* upsampleDepth (depth-maps.ts:9-42) */
__global__ void k_upsample_depth(const float* __restrict__ grid, int gw, int gh, int W, int H,
                                 float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H) return;
    const int x = i % W, y = i / W;
    const double gy = fmin((double)(gh - 1), fmax(0.0, ((y + 0.5) / H) * gh - 0.5));
    const int y0 = (int)floor(gy);
    const int y1 = min(gh - 1, y0 + 1);
    const double wy = gy - y0;
    const double gx = fmin((double)(gw - 1), fmax(0.0, ((x + 0.5) / W) * gw - 0.5));
    const int x0 = (int)floor(gx);
    const int x1 = min(gw - 1, x0 + 1);
    const double wx = gx - x0;
    const double d[4] = {grid[(size_t)y0 * gw + x0], grid[(size_t)y0 * gw + x1],
                         grid[(size_t)y1 * gw + x0], grid[(size_t)y1 * gw + x1]};
    const double w[4] = {(1 - wx) * (1 - wy), wx * (1 - wy), (1 - wx) * wy, wx * wy};
    double sum = 0.0, weight = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (d[k] > 0.0) {
            sum += d[k] * w[k];
            weight += w[k];
        }
    out[i] = weight > 0.5 ? (float)(sum / weight) : 0.0f;
}

inline unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }

inline bool on_words(const uint8_t* p) { return ((size_t)p & 3) == 0; }

/* Threads that fill the chip for gray bytes: a lane's load is one byte there, so lanes that are not needed to
 * fill it only split rows that one thread reads from the same sectors (4000 x 3000 to 500 x 375: eight lanes
 * 19.2 us, one 6.2; to 200 x 150: sixteen 20.5, four 11.3; 2^17 threads: 13.9). */
constexpr long long kGrayThreads = 1 << 16;

template <int KIND>
cudaError_t launch_blocks(const uint8_t* src, int W, int H, int tw, int th, uint8_t* out, cudaStream_t s) {
    const double sx = (double)W / tw, sy = (double)H / th;
    /* lanes per block: up to a warp, none without a pixel; blocks of less than eight columns are one
     * lane's (1280 x 960 to RGB means of 4 x 4: one lane 5.7 us, four 7.5; 8 x 8: 9.7, eight lanes 7.2) */
    int shift = 0;
    const long long pixels = (long long)tw * th;
    if (sx >= 8.0)
        while (shift < 5 && (2 << shift) <= sx && (KIND != BLOCK_GRAY || pixels << shift < kGrayThreads)) shift++;
    const long long threads = pixels << shift;
    const unsigned grid = (unsigned)((threads + 255) / 256);
    const bool words = KIND != BLOCK_GRAY && on_words(src);
    /* the largest block's sums (and twice its count times 256) fit 32 bits below 2^15 pixels */
    const bool wide = (sx + 1.0) * (sy + 1.0) >= 32768.0;
    constexpr bool RGBA = KIND != BLOCK_GRAY, ONE = KIND != BLOCK_RGB;
    auto* kernel = wide ? (words ? k_blocks<KIND, RGBA, true, false> : k_blocks<KIND, false, true, false>)
                   : shift ? (words ? k_blocks<KIND, RGBA, false, false> : k_blocks<KIND, false, false, false>)
                           : (words ? k_blocks<KIND, RGBA, false, ONE> : k_blocks<KIND, false, false, ONE>);
    kernel<<<grid, 256, 0, s>>>(src, W, H, tw, th, sx, sy, shift, out);
    return cudaGetLastError();
}

template <bool RGBA, bool WORDS>
cudaError_t launch_area(const uint8_t* src, int W, int H, int tw, int th, const L3dAreaCover& cols,
                        const L3dAreaCover& rows, float* temp, uint8_t* out, cudaStream_t s) {
    if (!temp) {
        const unsigned grid = ((unsigned)(tw + 31) / 32) * ((unsigned)(th + 7) / 8);
        if (cols.kmax <= 4 && rows.kmax <= 4)
            k_area<RGBA, WORDS, true><<<grid, dim3(32, 8), 0, s>>>(src, W, tw, th, cols, rows, out);
        else
            k_area<RGBA, WORDS, false><<<grid, dim3(32, 8), 0, s>>>(src, W, tw, th, cols, rows, out);
    } else {
        k_area_rows<RGBA, WORDS><<<blocks_for((long long)tw * H), 256, 0, s>>>(src, W, H, tw, cols, temp);
        k_area_cols<<<blocks_for((long long)tw * th), 256, 0, s>>>(temp, tw, th, rows, out);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t l3d_launch_gray_blocks(const uint8_t* rgba, int W, int H, int tw, int th, uint8_t* out,
                                   cudaStream_t s) {
    return launch_blocks<BLOCK_LUMA>(rgba, W, H, tw, th, out, s);
}
bool l3d_area_needs_temp(const L3dAreaCover& cols, const L3dAreaCover& rows, bool rgba, int tw, int th) {
    return cols.kmax > AREA_TAPS || rows.kmax > AREA_TAPS || (long long)tw * th > (rgba ? AREA_RGBA : AREA_GRAY);
}
cudaError_t l3d_launch_area(const uint8_t* src, bool rgba, int W, int H, int tw, int th,
                            const L3dAreaCover& cols, const L3dAreaCover& rows, float* temp,
                            uint8_t* out, cudaStream_t s) {
    if (!rgba) return launch_area<false, false>(src, W, H, tw, th, cols, rows, temp, out, s);
    if (on_words(src)) return launch_area<true, true>(src, W, H, tw, th, cols, rows, temp, out, s);
    return launch_area<true, false>(src, W, H, tw, th, cols, rows, temp, out, s);
}
cudaError_t l3d_launch_rgb_blocks(const uint8_t* rgba, int W, int H, int tw, int th, uint8_t* out,
                                  cudaStream_t s) {
    return launch_blocks<BLOCK_RGB>(rgba, W, H, tw, th, out, s);
}
cudaError_t l3d_launch_gray_down_blocks(const uint8_t* gray, int W, int H, int tw, int th, uint8_t* out,
                                        cudaStream_t s) {
    return launch_blocks<BLOCK_GRAY>(gray, W, H, tw, th, out, s);
}
cudaError_t l3d_launch_upsample_depth(const float* grid, int gw, int gh, int W, int H, float* out,
                                      cudaStream_t s) {
    k_upsample_depth<<<blocks_for((long long)W * H), 256, 0, s>>>(grid, gw, gh, W, H, out);
    return cudaGetLastError();
}

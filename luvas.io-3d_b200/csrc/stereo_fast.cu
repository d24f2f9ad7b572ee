/*
 * PatchMatch multi-view stereo, batched forms: every reference view of a batch in one launch
 * per kernel (init, each red/black colour, pack).
 *
 * Same algorithm, RNG stream and candidate schedule as frontend/src/app/vision/mvs/
 * patchmatch.wgsl.ts (init 255-289, propagate 349-423, pack 425-433).  Two evaluators of the
 * multi-view NCC share the kernels:
 *
 * Fast (L3D_FORM_FAST, mixed precision):
 *   - source images are FP16 (or FP32, U8) CUDA arrays read through the texture unit with
 *     hardware bilinear filtering at q.xy / q.z (the same filtered fetch the WGSL's
 *     textureSampleLevel does); BF16 storage is sampled from linear memory with FP32 weights;
 *   - the warped window is convex (q.z is affine and each image bound is a linear inequality in
 *     the reference pixel once multiplied by q.z > 0), so its four corner samples decide whether
 *     any of the 36 samples leaves the image: one test replaces 36 per-sample bounds checks and
 *     the sample loop runs branch-free with incremental homogeneous coordinates;
 *   - the NCC sums are accumulated in FP32 on values shifted by the reference window's centre
 *     pixel (the shifted-data form of the weighted variance, which removes the cancellation of
 *     E[x^2] - E[x]^2), with the reference terms w and w (r - c) precomputed per pixel;
 *     optionally compensated: FP32 row partials added with Neumaier compensation;
 *   - the k-best view mean keeps the three smallest costs in registers (same sum order as the
 *     reference's partial selection sort).
 *
 * Exact (L3D_FORM_EXACT): the plain form's arithmetic, operation for operation (per-sample
 * homogeneous coordinates, IEEE reciprocal, exact bilinear weights, raw-value sums, l3d_fmath.h
 * transcendentals), so a batched solve equals the plain per-view solve and the FP32 oracle bit
 * for bit.  Samples come from FP32 CUDA arrays through texture gathers: the four texels of a
 * bilinear footprint are fetched by one tld4 at the footprint's centre (integer coordinates
 * chosen in software, so the hardware's coordinate rounding cannot move the footprint) and
 * weighted in FP32 exactly as the oracle does.  With compensation on, every window sum is a
 * Neumaier sum (the oracle's compensated mode restates the same operations).
 *
 * Blocks are tiles of 16 x 8 pixels of one colour of one view; a block loads its view's
 * parameters (homography bases composed in FP64 on the host) into shared memory.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <cuda_fp16.h>

#include "l3d_fmath.h"
#include "l3d_internal.h"
#include "l3d_lanes.cuh"
#include "l3d_window.cuh"

namespace {

constexpr int TX = 16;   /* colour columns per tile */
constexpr int TY = 8;    /* rows per tile */
constexpr int S = 36;    /* 6 x 6 window, offsets -5, -3, ..., 5 */
/* How the propagate step is laid out for one evaluator: resident blocks per SM of the kernel with a
 * thread per pixel and of the one with eight lanes per pixel (l3d_lanes.cuh), and the largest launches,
 * in 128-pixel tiles of one colour, that take the lanes: with one source per view, two, and more.  What the
 * lanes do eight times over (random numbers, rays, the windows' sums) is done once per candidate however
 * many sources share it, so with few of them the thread per pixel wins earlier. */
struct Layout {
    int blocks, lane_blocks, lane_tiles[3];
};
/* Measured at 640x480, 8 sources, 3 iterations (ms, thread / lanes), 300, 675, 1200, 2400, 4800
 * tiles.  Filtered samples keep the texture pipe busy either way; the lanes win while the thread
 * kernel's last wave is a large part of it: 1.25 / 0.97, 2.36 / 2.04, 3.99 / 3.69, 7.69 / 7.57,
 * 15.7 / 15.8. */
constexpr Layout kFilter = {5, 5, {450, 1000, 3000}};
/* (FP16, 3 iterations, thread / lanes, one source: 300 tiles 0.37 / 0.37, 675 0.59 / 0.70, 1200 0.92 / 1.17;
 * two: 675 1.07 / 0.96, 1200 1.58 / 1.62, 2400 2.82 / 3.08; three: 2400 4.14 / 4.02.)  BF16 loads keep the
 * LSU busy instead: four sources 300 tiles 2.47 / 1.76, 675 3.84 / 3.79, 2400 13.4 / 13.6, 4800 25.4 / 27.5. */
constexpr Layout kLinear = {5, 5, {450, 1000, 1000}};
/* Gathers are bound by latency and issue; a quarter of the lanes idle in the lanes' second round:
 * 1.81 / 1.54, 4.00 / 3.24, 5.68 / 5.75. */
constexpr Layout kGather = {4, 5, {1000, 1000, 1000}};
/* The exact evaluator likewise: 2.13 / 1.72, 4.41 / 3.77, 6.47 / 6.81.  With four blocks the compiler
 * has the registers to keep a row's gathers in flight, which is worth more than warps (four views,
 * 5 iterations, thread per pixel: 3 blocks 35.6 ms, 4 35.9 ms, 5 38.9 ms). */
constexpr Layout kExact = {4, 4, {1000, 1000, 1000}};

__device__ __forceinline__ float dot3f(float3 a, float3 b) {
    return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x));
}
__device__ __forceinline__ float3 normalize_fast(float3 v) {
    float il = rsqrtf(dot3f(v, v));
    return make_float3(v.x * il, v.y * il, v.z * il);
}
/* normalize with an IEEE square root and reciprocal (the plain form's and oracle's order) */
__device__ __forceinline__ float3 normalize_ieee(float3 v) {
    float il = 1.0f / sqrtf(dot3f(v, v));
    return make_float3(v.x * il, v.y * il, v.z * il);
}
__device__ __forceinline__ float maxw(float a, float b) { return a > b ? a : b; }  /* WGSL max */
__device__ __forceinline__ float minw(float a, float b) { return a < b ? a : b; }

/* A running FP32 sum, plain (COMP = false: s += x, s = fma(a, b, s)) or Neumaier-compensated
 * (COMP = true): every addend, products rounded to FP32 first, goes through
 *   t = s + x;  c += |s| >= |x| ? (s - t) + x : (x - t) + s;  s = t,
 * and the sum is s + c.  The error of the compensated sum is bounded by about 2 ulp of the sum
 * of magnitudes independently of the number of terms (Neumaier 1974); the plain sum's bound
 * grows with the 36 terms of a window. */
template <bool COMP>
struct Acc {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x) {
        if (COMP) {
            const float t = s + x;
            const bool big = fabsf(s) >= fabsf(x);
            const float hi = big ? s : x, lo = big ? x : s;
            c = c + ((hi - t) + lo);
            s = t;
        } else {
            s = s + x;
        }
    }
    /* s + a * b: one fused multiply-add, or the rounded product added with compensation */
    __device__ __forceinline__ void fma_add(float a, float b) {
        if (COMP) add(a * b);
        else s = fmaf(a, b, s);
    }
    __device__ __forceinline__ float value() const { return COMP ? s + c : s; }
};

/* The three sums over a reference window's pairs (w, a): sum w, sum w a, sum w a^2. */
template <bool COMP>
struct RefSums {
    Acc<COMP> sw, sr, srr;
    __device__ __forceinline__ void add(float2 p) {
        sw.add(p.x);
        sr.fma_add(p.x, p.y);
        srr.fma_add(p.x * p.y, p.y);
    }
};

/* The three source-window sums of the fast evaluator (sum w s', sum w s'^2, sum w r' s' over
 * shifted values).  Plain (COMP = false): sequential FP32 sums in sample order.  Compensated:
 * each 6-sample window row is summed in FP32 (a row partial), and the row partials are added
 * with Neumaier compensation; the rounding error is then bounded by about 7 ulp of the sum of
 * magnitudes instead of 35 for the sequential sum, at 7 extra operations per row and sum
 * instead of per sample (the fast propagate kernel is bound by the texture pipe, not by issue,
 * so the row-level compensation costs it next to nothing; per-sample compensation did). */
template <bool COMP>
struct WinSums {
    Acc<COMP> ss, sss, srs;
    float rs = 0.0f, rss = 0.0f, rrs = 0.0f;
    __device__ __forceinline__ void term(float t, float sv, float rwr) {
        if (COMP) {
            rs = rs + t;
            rss = fmaf(t, sv, rss);
            rrs = fmaf(rwr, sv, rrs);
        } else {
            ss.s = ss.s + t;
            sss.s = fmaf(t, sv, sss.s);
            srs.s = fmaf(rwr, sv, srs.s);
        }
    }
    __device__ __forceinline__ void end_row() {
        if (COMP) {
            ss.add(rs);
            sss.add(rss);
            srs.add(rrs);
            rs = rss = rrs = 0.0f;
        }
    }
};

__device__ __forceinline__ float unpack_depth(uint32_t packed) {
    return l3d_f16_to_f32(packed & 0xffffu);
}
/* unpack_normal of depth-packing.wgsl.ts:3-19 in the plain form's operation order */
__device__ __forceinline__ float3 unpack_normal_ieee(uint32_t packed) {
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
    return normalize_ieee(n);
}
__device__ __forceinline__ float3 unpack_normal(uint32_t packed) {
    float ex = (float)((packed >> 16) & 63u) * (2.0f / 63.0f) - 1.0f;
    float ey = (float)((packed >> 22) & 63u) * (2.0f / 63.0f) - 1.0f;
    float3 n = make_float3(ex, ey, (1.0f - fabsf(ex)) - fabsf(ey));
    if (n.z < 0.0f) {
        float nx = (1.0f - fabsf(n.y)) * (n.x >= 0.0f ? 1.0f : -1.0f);
        float ny = (1.0f - fabsf(n.x)) * (n.y >= 0.0f ? 1.0f : -1.0f);
        n.x = nx;
        n.y = ny;
    }
    return normalize_fast(n);
}
__device__ __forceinline__ uint32_t pack_sample(float depth, float3 n, float cost) {
    if (!(depth > 0.0f) || !(cost < 1.0f)) return 0u;
    float s = (fabsf(n.x) + fabsf(n.y)) + fabsf(n.z);
    float ex = n.x / s, ey = n.y / s;
    if (n.z < 0.0f) {
        float nx = (1.0f - fabsf(ey)) * (ex >= 0.0f ? 1.0f : -1.0f);
        float ny = (1.0f - fabsf(ex)) * (ey >= 0.0f ? 1.0f : -1.0f);
        ex = nx;
        ey = ny;
    }
    float cx = fminf(fmaxf(fmaf(ex, 0.5f, 0.5f), 0.0f), 1.0f);
    float cy = fminf(fmaxf(fmaf(ey, 0.5f, 0.5f), 0.0f), 1.0f);
    uint32_t qx = (uint32_t)fmaf(cx, 63.0f, 0.5f);
    uint32_t qy = (uint32_t)fmaf(cy, 63.0f, 0.5f);
    uint32_t c = min(15u, (uint32_t)(cost * 15.0f));
    return (l3d_f32_to_f16(depth) & 0xffffu) | (qx << 16) | (qy << 22) | (c << 28);
}

/* The four texels of the bilinear footprint whose top-left texel is (x0, y0), from a texture
 * gather (tld4) at the footprint's centre: in unnormalised coordinates the centre of texel i is
 * i + 0.5, so coordinate x0 + 1 lies exactly between texels x0 and x0 + 1 and the footprint
 * cannot shift with the texture unit's coordinate rounding.  Clamp addressing repeats the last
 * row and column like the oracle's min(i + 1, size - 1).  The gather returns the footprint as
 * (x0, y0+1), (x0+1, y0+1), (x0+1, y0), (x0, y0) in x, y, z, w. */
__device__ __forceinline__ float bilinear_gather(unsigned long long tex, float u, float v) {
    const float x0 = floorf(u), y0 = floorf(v);
    const float fx = u - x0, fy = v - y0;
    const float4 g = tex2Dgather<float4>((cudaTextureObject_t)tex, x0 + 1.0f, y0 + 1.0f, 0);
    const float a = g.w, b = g.z, c = g.x, e = g.y;
    const float top = fmaf(fx, b - a, a);
    const float bot = fmaf(fx, e - c, c);
    return fmaf(fy, bot - top, top);
}

/* Image access: texture path (F16/F32 CUDA arrays, hardware bilinear) or BF16 linear memory. */
template <bool TEX>
struct Img {
    /* value at filtering coordinate (u, v) = texel coordinate + 0.5 */
    static __device__ __forceinline__ float sample(unsigned long long tex, const uint16_t* img,
                                                   int W, int H, float u, float v) {
        if (TEX) {
            return tex2D<float>((cudaTextureObject_t)tex, u, v);
        } else {
            float x = u - 0.5f, y = v - 0.5f;
            float x0 = floorf(x), y0 = floorf(y);
            float fx = x - x0, fy = y - y0;
            int ix0 = min(max((int)x0, 0), W - 1), iy0 = min(max((int)y0, 0), H - 1);
            int ix1 = min(ix0 + 1, W - 1), iy1 = min(iy0 + 1, H - 1);
            const uint16_t* r0 = img + (long long)iy0 * W;
            const uint16_t* r1 = img + (long long)iy1 * W;
            float a = __uint_as_float((uint32_t)__ldg(r0 + ix0) << 16);
            float b = __uint_as_float((uint32_t)__ldg(r0 + ix1) << 16);
            float c = __uint_as_float((uint32_t)__ldg(r1 + ix0) << 16);
            float e = __uint_as_float((uint32_t)__ldg(r1 + ix1) << 16);
            float top = fmaf(fx, b - a, a);
            float bot = fmaf(fx, e - c, c);
            return fmaf(fy, bot - top, top);
        }
    }
    static __device__ __forceinline__ float texel(unsigned long long tex, const uint16_t* img,
                                                  int W, int H, int x, int y) {
        if (TEX) {
            return tex2D<float>((cudaTextureObject_t)tex, (float)x + 0.5f, (float)y + 0.5f);
        } else {
            x = min(max(x, 0), W - 1);
            y = min(max(y, 0), H - 1);
            return __uint_as_float((uint32_t)__ldg(img + (long long)y * W + x) << 16);
        }
    }
};

/* Software bilinear sample from the pair image (each texel stores itself and its right
 * neighbour as half2), at filtering coordinate (u, v): two 32-bit loads on the LSU path, FP32
 * weights.  Used for the window rows the texture unit does not take. */
__device__ __forceinline__ float pair_sample(const uint32_t* __restrict__ pairs, int W, int H,
                                             float u, float v) {
    float x = u - 0.5f, y = v - 0.5f;
    int x0 = __float2int_rd(x), y0 = __float2int_rd(y);
    float fx = x - (float)x0, fy = y - (float)y0;
    x0 = min(max(x0, 0), W - 1);
    y0 = min(max(y0, 0), H - 1);
    int y1 = min(y0 + 1, H - 1);
    uint32_t t = __ldg(pairs + (long long)y0 * W + x0);
    uint32_t b = __ldg(pairs + (long long)y1 * W + x0);
    float2 tf = __half22float2(*reinterpret_cast<const __half2*>(&t));
    float2 bf = __half22float2(*reinterpret_cast<const __half2*>(&b));
    float top = fmaf(fx, tf.y - tf.x, tf.x);
    float bot = fmaf(fx, bf.y - bf.x, bf.x);
    return fmaf(fy, bot - top, top);
}

/* reproject (patchmatch.wgsl.ts:166-190): the reference point x seen from source sv, rounded to
 * a source pixel, back-projected with that pixel's packed depth; false when any step fails.
 * Operation order of the plain form. */
__device__ __forceinline__ bool reproject(const L3dFastView& v, const L3dFastDev& d,
                                          const L3dFastSrc& sv, float px, float py, float3 x,
                                          float* dist, float* z) {
    const float* R = sv.R;
    float3 xs = make_float3(fmaf(R[2], x.z, fmaf(R[1], x.y, fmaf(R[0], x.x, sv.t[0]))),
                            fmaf(R[5], x.z, fmaf(R[4], x.y, fmaf(R[3], x.x, sv.t[1]))),
                            fmaf(R[8], x.z, fmaf(R[7], x.y, fmaf(R[6], x.x, sv.t[2]))));
    if (!(xs.z > 1e-6f)) return false;
    float iz = 1.0f / xs.z;
    float rx = rintf(fmaf(sv.k[0] * xs.x, iz, sv.k[2]));
    float ry = rintf(fmaf(sv.k[1] * xs.y, iz, sv.k[3]));
    if (!(rx >= 0.0f && ry >= 0.0f && rx < (float)sv.W && ry < (float)sv.H)) return false;
    uint32_t packed = __ldg(d.depths + sv.dep_off + (long long)(int)ry * sv.W + (int)rx);
    float ds = unpack_depth(packed);
    if (!(ds > 0.0f) || (packed >> 28) > L3D_FILTER_COST) return false;
    float3 e = make_float3(((rx - sv.k[2]) / sv.k[0]) * ds - sv.t[0],
                           ((ry - sv.k[3]) / sv.k[1]) * ds - sv.t[1], ds - sv.t[2]);
    float3 back = make_float3(fmaf(R[6], e.z, fmaf(R[3], e.y, R[0] * e.x)),
                              fmaf(R[7], e.z, fmaf(R[4], e.y, R[1] * e.x)),
                              fmaf(R[8], e.z, fmaf(R[5], e.y, R[2] * e.x)));
    if (!(back.z > 1e-6f)) return false;
    float bz = 1.0f / back.z;
    float dx = fmaf(v.k[0] * back.x, bz, v.k[2]) - px;
    float dy = fmaf(v.k[1] * back.y, bz, v.k[3]) - py;
    *dist = sqrtf(fmaf(dx, dx, dy * dy));
    *z = back.z;
    return true;
}

/* hypothesis_cost (patchmatch.wgsl.ts:192-233) over evaluator E's view_cost: range and
 * orientation tests, u = (K_r^-T n) / rho, per-source cost (+ geometric term), mean of the
 * k = max(1, min(3, S - 1)) smallest.  The three smallest are kept in registers, ascending; the
 * reference's partial selection sort adds the same values in the same order. */
template <class E, class P>
__device__ __forceinline__ float hyp_cost(const E& e, const L3dFastView& v, const L3dFastDev& d,
                                          const P& s, float3 n, float dd) {
    if (!(dd > 0.0f)) return 2.0f;
    float inv = 1.0f / dd;
    if (inv > v.range[0] || inv < v.range[1]) return 2.0f;
    if (dot3f(n, s.ray) >= -1e-3f) return 2.0f;
    const int count = v.n;
    if (count == 0) return 2.0f;
    float3 x = make_float3(s.ray.x * dd, s.ray.y * dd, dd);
    float ir = 1.0f / dot3f(n, x);
    float u[3];
    u[0] = (n.x * v.kinv[0]) * ir;
    u[1] = (n.y * v.kinv[1]) * ir;
    u[2] = fmaf(n.x, v.kinv[2], fmaf(n.y, v.kinv[3], n.z)) * ir;
    const bool geometric = (v.flags & 1u) != 0u;
    float b0 = 3.0e38f, b1 = 3.0e38f, b2 = 3.0e38f;
    for (int k = 0; k < count; k++) {
        float c = e.view_cost(s, v.src[k], u);
        if (geometric) {
            float dist, z;
            bool ok = reproject(v, d, v.src[k], s.px, s.py, x, &dist, &z);
            c = fmaf(v.range[3], ok ? minw(dist, 3.0f) : 3.0f, c);
        }
        if (c < b2) {
            if (c < b1) {
                b2 = b1;
                if (c < b0) {
                    b1 = b0;
                    b0 = c;
                } else {
                    b1 = c;
                }
            } else {
                b2 = c;
            }
        }
    }
    const int kk = max(1, min(3, count - 1));
    float total = b0;
    if (kk > 1) total = total + b1;
    if (kk > 2) total = total + b2;
    return total / (float)kk;
}

/* One pixel's reference window in shared memory: 36 pairs of window values, pair i at
 * win[i * STRIDE].  k_fast_propagate_lanes keeps a pixel's pairs together (STRIDE 1: the eight lanes
 * of a pixel read the same pair, a broadcast); the kernels with one thread per pixel, k_fast_propagate
 * among them, keep a column per thread (STRIDE 128: consecutive threads read consecutive pairs).  The exact evaluator's pairs
 * are (w, r), the fast evaluator's (w, w (r - c)), c the centre pixel. */
constexpr int XBLOCK = 128;

/* Per-pixel state of the fast evaluator. */
template <int STRIDE>
struct FPix {
    static constexpr int kStride = STRIDE;
    const float2* win;
    float center, inv_sum, mean_r, var_r;
    uint32_t rng;
    float px, py;
    float3 ray;
};

/* What the evaluators share: the view and the buffers, rays and random depths. */
struct Scene {
    const L3dFastView& v;
    const L3dFastDev& d;
    __device__ Scene(const L3dFastView& view, const L3dFastDev& dev) : v(view), d(dev) {}

    static __device__ __forceinline__ float dot(float3 a, float3 b) { return dot3f(a, b); }
    __device__ float3 ray_of(float x, float y) const {
        return make_float3((x - v.k[2]) / v.k[0], (y - v.k[3]) / v.k[1], 1.0f);
    }
    /* random_depth (patchmatch.wgsl.ts:243-249) */
    template <class P>
    __device__ float random_depth(P& s) const {
        float t = l3d_random(&s.rng);
        return 1.0f / fmaf(v.range[0], t, v.range[1] * (1.0f - t));
    }
    /* The pixel's RNG state, coordinates and ray (seed, patchmatch.wgsl.ts:251-253). */
    template <class P>
    __device__ void begin(P& s, int x, int y, int iteration, int phase) const {
        s.px = (float)x;
        s.py = (float)y;
        uint32_t seed = (uint32_t)(v.ref + 1) * 0x9e3779b1u + (uint32_t)iteration * 97u +
                        (uint32_t)phase * 13u + (v.flags & 1u) * 7u;
        s.rng = l3d_pcg((uint32_t)(y * v.W + x) ^
                        l3d_pcg(seed + (uint32_t)iteration * 7919u + (uint32_t)phase * 104729u));
        s.ray = ray_of(s.px, s.py);
    }
};

/* TEX: texture-unit sampling of F16/F32 arrays (false: BF16 linear memory).  TEXROWS: window
 * rows (of 6) sampled by the texture unit; the other rows use pair_sample (TEX only).  COMP:
 * compensated window sums.  GATHER: the texture rows are texture gathers weighted with exact
 * FP32 bilinear weights instead of hardware-filtered fetches (8-bit weights). */
template <bool TEX, int TEXROWS = 6, bool COMP = false, bool GATHER = false>
struct Fast : Scene {
    template <int STRIDE> using Pix = FPix<STRIDE>;
    static constexpr Layout kLayout = GATHER ? kGather : TEX ? kFilter : kLinear;
    /* window rows unrolled together: filtered samples want all their fetches in flight, a gather's
     * row of blends is long enough that more than two overflow the instruction cache (four views of
     * 640x480, 8 sources, 5 iterations: 33.6 ms, all six rows 34.6; filtered 23.9 and 23.6) */
    static constexpr int kRows = GATHER ? 2 : 6;
    using Scene::Scene;

    static __device__ __forceinline__ float3 normalize(float3 a) { return normalize_fast(a); }
    static __device__ __forceinline__ float3 unpack_n(uint32_t packed) { return unpack_normal(packed); }

    __device__ const uint16_t* img(long long off) const {
        return (const uint16_t*)d.images + off;
    }

    /* prepare_window (patchmatch.wgsl.ts:90-110), shifted by the centre pixel, in three steps so
     * that the lanes of a pixel can share the first: the centre, pair i as (w, r - c), and the
     * sums in sample order; scale() turns a pair into the stored (w, w (r - c)). */
    __device__ float center(int x, int y) const {
        return Img<TEX>::texel(v.ref_tex, img(v.ref_img_off), v.W, v.H, x, y);
    }
    __device__ float2 pair(int x, int y, int i, float c) const {
        const float ic1 = 1.0f / (2.0f * 0.06f * 0.06f);
        const int ox = (i % 6) * 2 - 5, oy = (i / 6) * 2 - 5;
        const float spatial = (float)(ox * ox + oy * oy) / (2.0f * 5.0f * 5.0f);
        const float val = Img<TEX>::texel(v.ref_tex, img(v.ref_img_off), v.W, v.H, x + ox, y + oy);
        const float dc = val - c;
        return make_float2(__expf(-(dc * dc) * ic1 - spatial), dc);
    }
    using Sums = RefSums<COMP>;
    template <class P>
    __device__ void finish(P& s, const Sums& m, float c) const {
        s.center = c;
        s.inv_sum = 1.0f / m.sw.value();
        s.mean_r = m.sr.value() * s.inv_sum;
        s.var_r = fmaxf(fmaf(-s.mean_r, s.mean_r, m.srr.value() * s.inv_sum), 0.0f);
    }
    static __device__ __forceinline__ float2 scale(float2 p) { return make_float2(p.x, p.x * p.y); }

    /* one sample's terms of the window sums: w s', s' and (w r') s' (s' = s - c, r' = r - c) */
    template <class P>
    static __device__ __forceinline__ void window_term(WinSums<COMP>& ws, const P& s, int i, float sv) {
        const float2 w = s.win[i * P::kStride];
        ws.term(w.x * sv, sv, w.y);
    }

    /* view_cost (patchmatch.wgsl.ts:130-159) with H = Bt + ktt u^T. */
    template <class P>
    __device__ float view_cost(const P& s, const L3dFastSrc& src, const float* u) const {
        float h[9];
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int c = 0; c < 3; c++) h[r * 3 + c] = fmaf(src.ktt[r], u[c], src.Bt[r * 3 + c]);
        const float x0 = s.px - 5.0f, y0 = s.py - 5.0f;
        /* q at the window's top-left sample and its steps along x and y (2 pixels) */
        const float qx0 = fmaf(h[0], x0, fmaf(h[1], y0, h[2]));
        const float qy0 = fmaf(h[3], x0, fmaf(h[4], y0, h[5]));
        const float qz0 = fmaf(h[6], x0, fmaf(h[7], y0, h[8]));
        const float dxx = 2.0f * h[0], dxy = 2.0f * h[3], dxz = 2.0f * h[6];
        const float dyx = 2.0f * h[1], dyy = 2.0f * h[4], dyz = 2.0f * h[7];
        /* the four corner samples decide validity for the whole (convex) window */
        const float umax = (float)src.W - 0.5f, vmax = (float)src.H - 0.5f;
        bool ok = true;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float fx = (c & 1) ? 5.0f : 0.0f, fy = (c & 2) ? 5.0f : 0.0f;
            float qz = fmaf(dyz, fy, fmaf(dxz, fx, qz0));
            float qx = fmaf(dyx, fy, fmaf(dxx, fx, qx0));
            float qy = fmaf(dyy, fy, fmaf(dxy, fx, qy0));
            ok = ok && qz > 1e-6f && qx >= 0.5f * qz && qy >= 0.5f * qz && qx <= umax * qz &&
                 qy <= vmax * qz;
        }
        if (!ok) return 2.0f;
        const uint16_t* si = img(src.img_off);
        WinSums<COMP> ws;
        /* rows [0, TEXROWS) through the texture unit, rows [TEXROWS, 6) through pair_sample: two
         * loops with constant bounds, so each unrolls into straight-line code with all its
         * fetches in flight together */
        constexpr int RT = TEX ? TEXROWS : 6;
        float rx = qx0, ry = qy0, rz = qz0;
#pragma unroll kRows
        for (int r = 0; r < RT; r++) {
            float qx = rx, qy = ry, qz = rz;
#pragma unroll
            for (int c = 0; c < 6; c++) {
                const int i = r * 6 + c;
                float iz = l3d_rcp_approx(qz);
                float val = GATHER ? bilinear_gather(src.tex, fmaf(qx, iz, -0.5f), fmaf(qy, iz, -0.5f))
                                   : Img<TEX>::sample(src.tex, si, src.W, src.H, qx * iz, qy * iz);
                float sv = val - s.center;
                window_term(ws, s, i, sv);
                qx += dxx;
                qy += dxy;
                qz += dxz;
            }
            ws.end_row();
            rx += dyx;
            ry += dyy;
            rz += dyz;
        }
        if constexpr (TEX && TEXROWS < 6) {
            const uint32_t* sp = d.pairs + src.img_off;
#pragma unroll
            for (int r = TEXROWS; r < 6; r++) {
                float qx = rx, qy = ry, qz = rz;
#pragma unroll
                for (int c = 0; c < 6; c++) {
                    const int i = r * 6 + c;
                    float iz = l3d_rcp_approx(qz);
                    float val = pair_sample(sp, src.W, src.H, qx * iz, qy * iz);
                    float sv = val - s.center;
                    window_term(ws, s, i, sv);
                    qx += dxx;
                    qy += dxy;
                    qz += dxz;
                }
                ws.end_row();
                rx += dyx;
                ry += dyy;
                rz += dyz;
            }
        }
        float mean = ws.ss.value() * s.inv_sum;
        float var_s = fmaxf(fmaf(-mean, mean, ws.sss.value() * s.inv_sum), 0.0f);
        float prod = s.var_r * var_s;
        if (prod < 1e-10f) return 1.0f;  /* sqrt(prod) < 1e-5 */
        float cov = fmaf(-s.mean_r, mean, ws.srs.value() * s.inv_sum);
        return fminf(fmaxf(1.0f - cov * rsqrtf(prod), 0.0f), 2.0f);
    }

    /* hypothesis_cost (patchmatch.wgsl.ts:192-233) */
    template <class P>
    __device__ float cost_of(const P& s, float3 n, float dd) const {
        return hyp_cost(*this, v, d, s, n, dd);
    }

    /* random_normal (patchmatch.wgsl.ts:235-242) */
    template <class P>
    __device__ float3 random_normal(P& s) const {
        float z = fmaf(l3d_random(&s.rng), 2.0f, -1.0f);
        float a = l3d_random(&s.rng) * 6.2831853f;
        float r = sqrtf(fmaxf(0.0f, fmaf(-z, z, 1.0f)));
        float sn, cs;
        __sincosf(a, &sn, &cs);
        float3 n = make_float3(r * cs, r * sn, z);
        float3 view = normalize_fast(s.ray);
        if (dot3f(n, view) > 0.0f) n = make_float3(-n.x, -n.y, -n.z);
        return normalize_fast(make_float3(fmaf(view.x, -0.5f, n.x), fmaf(view.y, -0.5f, n.y),
                                          fmaf(view.z, -0.5f, n.z)));
    }
};

/* Per-pixel state of the exact evaluator: the private block of patchmatch.wgsl.ts:49-54. */
template <int STRIDE>
struct XPix {
    static constexpr int kStride = STRIDE;
    const float2* win;
    float rsum, rmean, rvar;
    uint32_t rng;
    float px, py;
    float3 ray;
};

/* The plain form's arithmetic in the batched kernels (see the file header).  COMP: Neumaier-
 * compensated window sums (the oracle's compensated mode). */
template <bool COMP>
struct Exact : Scene {
    template <int STRIDE> using Pix = XPix<STRIDE>;
    static constexpr Layout kLayout = kExact;
    using Scene::Scene;

    static __device__ __forceinline__ float3 normalize(float3 a) { return normalize_ieee(a); }
    static __device__ __forceinline__ float3 unpack_n(uint32_t packed) { return unpack_normal_ieee(packed); }

    __device__ float ref_pixel(int x, int y) const {
        x = min(max(x, 0), v.W - 1);
        y = min(max(y, 0), v.H - 1);
        return __ldg((const float*)d.images + v.ref_img_off + (long long)y * v.W + x);
    }

    /* prepare_window (patchmatch.wgsl.ts:90-110), split like the fast evaluator's */
    __device__ float center(int x, int y) const { return ref_pixel(x, y); }
    __device__ float2 pair(int x, int y, int i, float c) const {
        const float c1 = 2.0f * 0.06f * 0.06f;
        const float c2 = 2.0f * 5.0f * 5.0f;
        const int ox = (i % 6) * 2 - 5, oy = (i / 6) * 2 - 5;
        const float val = ref_pixel(x + ox, y + oy);
        const float dc = val - c;
        return make_float2(l3d_expf(-(dc * dc) / c1 - (float)(ox * ox + oy * oy) / c2), val);
    }
    using Sums = RefSums<COMP>;
    template <class P>
    __device__ void finish(P& s, const Sums& m, float) const {
        s.rsum = m.sw.value();
        s.rmean = m.sr.value() / s.rsum;
        s.rvar = maxw(fmaf(-s.rmean, s.rmean, m.srr.value() / s.rsum), 0.0f);
    }
    static __device__ __forceinline__ float2 scale(float2 p) { return p; }

    /* The window sums of one source, every sample's position tested like the oracle does; false
     * when one is behind the camera or outside the image.  A rolled loop: only windows that graze an
     * image border (or leave the normal numbers) come here. */
    template <class P>
    __device__ bool sums_tested(const P& s, const L3dFastSrc& src, const float* h, Acc<COMP>& ss,
                                Acc<COMP>& sss, Acc<COMP>& srs) const {
        const float wmax = (float)(src.W - 1), hmax = (float)(src.H - 1);
#pragma unroll 1
        for (int i = 0; i < S; i++) {
            const float x = s.px + (float)((i % 6) * 2 - 5), y = s.py + (float)((i / 6) * 2 - 5);
            const float qz = fmaf(h[6], x, fmaf(h[7], y, h[8]));
            const float qx = fmaf(h[0], x, fmaf(h[1], y, h[2]));
            const float qy = fmaf(h[3], x, fmaf(h[4], y, h[5]));
            const float iz = 1.0f / qz;
            const float uu = qx * iz, vv = qy * iz;
            if (!(qz > 1e-6f) || !(uu >= 0.0f && vv >= 0.0f && uu <= wmax && vv <= hmax)) return false;
            const float val = bilinear_gather(src.tex, uu, vv);
            const float2 rwv = s.win[i * P::kStride];
            ss.fma_add(rwv.x, val);
            const float wv = rwv.x * val;
            sss.fma_add(wv, val);
            srs.fma_add(wv, rwv.y);
        }
        return true;
    }

    /* view_cost (patchmatch.wgsl.ts:130-159) with H = B + kt u^T (Bt/ktt hold the unshifted
     * base in this form).  Every sample is computed as the oracle computes it; a sample with
     * q.z <= 1e-6 or outside [0, W-1] x [0, H-1] makes the cost 2 (l3d_window.cuh).  Bound by latency
     * and issue: a test and a general division per sample, each a branch that cuts a row's gathers
     * apart, took 75.6 ms for four views of 640x480 (8 sources, 5 iterations); the straight line for
     * windows inside the image takes 35.9 ms. */
    template <class P>
    __device__ float view_cost(const P& s, const L3dFastSrc& src, const float* u) const {
        float h[9];
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int c = 0; c < 3; c++) h[r * 3 + c] = fmaf(src.ktt[r], u[c], src.Bt[r * 3 + c]);
        const L3dPlace place =
            l3d_window_place(h, s.px, s.py, 5.0f, (float)(src.W - 1), (float)(src.H - 1));
        Acc<COMP> ss, sss, srs;
        if (place == L3D_INSIDE) {
            /* rows rolled: unrolled they overflow the instruction cache (35.9 against 38.8 ms) */
#pragma unroll 1
            for (int r = 0; r < 6; r++) {
                const float y = s.py + (float)(r * 2 - 5);
                const float hz = fmaf(h[7], y, h[8]);
                const float hx = fmaf(h[1], y, h[2]);
                const float hy = fmaf(h[4], y, h[5]);
#pragma unroll
                for (int c = 0; c < 6; c++) {
                    const int i = r * 6 + c;
                    const float x = s.px + (float)(c * 2 - 5);
                    const float iz = l3d_rcp_normal(fmaf(h[6], x, hz));
                    const float val = bilinear_gather(src.tex, fmaf(h[0], x, hx) * iz, fmaf(h[3], x, hy) * iz);
                    const float2 rwv = s.win[i * P::kStride];
                    const float w = rwv.x;
                    ss.fma_add(w, val);
                    const float wv = w * val;
                    sss.fma_add(wv, val);
                    srs.fma_add(wv, rwv.y);
                }
            }
        } else if (place == L3D_OUTSIDE || !sums_tested(s, src, h, ss, sss, srs)) {
            return 2.0f;
        }
        const float mean = ss.value() / s.rsum;
        const float var_s = maxw(fmaf(-mean, mean, sss.value() / s.rsum), 0.0f);
        const float den = sqrtf(s.rvar * var_s);
        if (den < 1e-5f) return 1.0f;
        const float cov = fmaf(-s.rmean, mean, srs.value() / s.rsum);
        return minw(maxw(1.0f - cov / den, 0.0f), 2.0f);
    }

    /* hypothesis_cost (patchmatch.wgsl.ts:192-233) */
    template <class P>
    __device__ float cost_of(const P& s, float3 n, float dd) const {
        return hyp_cost(*this, v, d, s, n, dd);
    }

    /* random_normal (patchmatch.wgsl.ts:235-242) */
    template <class P>
    __device__ float3 random_normal(P& s) const {
        float z = fmaf(l3d_random(&s.rng), 2.0f, -1.0f);
        float a = l3d_random(&s.rng) * 6.2831853f;
        float r = sqrtf(maxw(0.0f, fmaf(-z, z, 1.0f)));
        float sn, cs;
        l3d_sincosf(a, &sn, &cs);
        float3 n = make_float3(r * cs, r * sn, z);
        float3 view = normalize_ieee(s.ray);
        if (dot3f(n, view) > 0.0f) n = make_float3(-n.x, -n.y, -n.z);
        return normalize_ieee(make_float3(fmaf(view.x, -0.5f, n.x), fmaf(view.y, -0.5f, n.y),
                                          fmaf(view.z, -0.5f, n.z)));
    }
};

/* The whole window of one pixel by one thread, in its column. */
template <class E>
__device__ __forceinline__ void thread_window(const E& f, typename E::template Pix<XBLOCK>& s, float2* win,
                                              int x, int y) {
    const float c = f.center(x, y);
    typename E::Sums sums;
#pragma unroll
    for (int i = 0; i < S; i++) {
        const float2 p = f.pair(x, y, i, c);
        sums.add(p);
        win[i * XBLOCK] = E::scale(p);
    }
    s.win = win;
    f.finish(s, sums, c);
}

/* Block -> (view, tile) and the view's parameters in shared memory. */
__device__ __forceinline__ int find_view(const L3dFastDev& d, int tile) {
    int lo = 0, hi = d.n_views - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(d.tile_start + mid) <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

/* The view table has an 8-byte aligned stride (static_assert below), so it is copied in 8-byte
 * words. */
static_assert(sizeof(L3dFastView) % 8 == 0, "view table stride must be a multiple of 8 bytes");
static_assert(alignof(L3dFastView) >= 8, "view table must be 8-byte aligned");
__device__ __forceinline__ void load_view(L3dFastView& dst, const L3dFastView* src) {
    const unsigned long long* s = (const unsigned long long*)src;
    unsigned long long* o = (unsigned long long*)&dst;
    for (int i = threadIdx.x; i < (int)(sizeof(L3dFastView) / 8); i += blockDim.x) o[i] = __ldg(s + i);
    __syncthreads();
}

template <class E>
__global__ void __launch_bounds__(128) k_fast_init(const L3dFastDev d) {
    __shared__ __align__(16) L3dFastView sv;
    __shared__ float2 windows[S * XBLOCK];
    load_view(sv, d.views + find_view(d, blockIdx.x));
    const int local = blockIdx.x - sv.tile_start;
    const int y = (local / sv.tiles_x) * TY + threadIdx.x / TX;
    /* init covers every pixel: a tile spans 32 image columns, two pixels per thread */
    E f(sv, d);
    for (int half = 0; half < 2; half++) {
        const int xx = (local % sv.tiles_x) * (2 * TX) + (threadIdx.x % TX) * 2 + half;
        if (xx >= sv.W || y >= sv.H) continue;
        typename E::template Pix<XBLOCK> s;
        f.begin(s, xx, y, 0, 0);
        thread_window(f, s, windows + threadIdx.x, xx, y);
        const long long index = (long long)y * sv.W + xx;
        float3 n = f.random_normal(s);
        float dd = f.random_depth(s);
        if (sv.has_coarse && d.coarse) {
            /* init_coarse (patchmatch.wgsl.ts:296-333): the random plane against the planes of
             * the four nearest coarse pixels, re-intersected with this pixel's ray */
            float c = f.cost_of(s, n, dd);
            const float qx = ((s.px + 0.5f) * (float)sv.cW) / (float)sv.W - 0.5f;
            const float qy = ((s.py + 0.5f) * (float)sv.cH) / (float)sv.H - 0.5f;
            const int bx = (int)floorf(qx), by = (int)floorf(qy);
            for (int corner = 0; corner < 4; corner++) {
                const int cx = min(max(bx + (corner & 1), 0), sv.cW - 1);
                const int cy = min(max(by + (corner >> 1), 0), sv.cH - 1);
                const float4 h = d.coarse[sv.coarse_off + (long long)cy * sv.cW + cx];
                if (!(h.w > 0.0f)) continue;
                const float3 hn = make_float3(h.x, h.y, h.z);
                const float3 point = make_float3(((float)cx - sv.ck[2]) / sv.ck[0] * h.w,
                                                 ((float)cy - sv.ck[3]) / sv.ck[1] * h.w, h.w);
                const float den = dot3f(hn, s.ray);
                if (fabsf(den) < 1e-6f) continue;
                const float hd = dot3f(hn, point) / den;
                const float hc = f.cost_of(s, hn, hd);
                if (hc < c) {
                    c = hc;
                    n = hn;
                    dd = hd;
                }
            }
            d.hyp[sv.pix_off + index] = make_float4(n.x, n.y, n.z, dd);
            d.cost[sv.pix_off + index] = c;
            continue;
        }
        if (sv.flags & 1u) {
            uint32_t packed = d.depths[sv.ref_dep_off + index];
            if (unpack_depth(packed) > 0.0f) {
                dd = unpack_depth(packed);
                n = E::unpack_n(packed);
            }
        }
        float c = f.cost_of(s, n, dd);
        if (!(sv.flags & 1u) && sv.has_prior) {
            float pd = d.prior[sv.pix_off + index];
            if (pd > 0.0f) {
                float3 vv = E::normalize(s.ray);
                float3 pn = make_float3(-vv.x, -vv.y, -vv.z);
                float pc = f.cost_of(s, pn, pd);
                if (pc < c) {
                    c = pc;
                    n = pn;
                    dd = pd;
                }
            }
        }
        d.hyp[sv.pix_off + index] = make_float4(n.x, n.y, n.z, dd);
        d.cost[sv.pix_off + index] = c;
    }
}

/* propagate (patchmatch.wgsl.ts:349-423), one thread per pixel; the four lanes of each hardware quad
 * take a 2 x 2 block of this colour's pixels (tighter texture footprints per quad request). */
template <class E>
__global__ void __launch_bounds__(128, E::kLayout.blocks) k_fast_propagate(const L3dFastDev d, int iteration,
                                                                           int phase, float step) {
    __shared__ __align__(16) L3dFastView sv;
    __shared__ float2 windows[S * XBLOCK];
    load_view(sv, d.views + find_view(d, blockIdx.x));
    if (iteration >= sv.iterations) return;
    const int local = blockIdx.x - sv.tile_start;
    const int q = threadIdx.x >> 2, j = threadIdx.x & 3;
    const int tx = (q % (TX / 2)) * 2 + (j & 1), ty = (q / (TX / 2)) * 2 + (j >> 1);
    const int y = (local / sv.tiles_x) * TY + ty;
    const int x = ((local % sv.tiles_x) * TX + tx) * 2 + ((y + phase) & 1);
    if (x >= sv.W || y >= sv.H) return;
    E f(sv, d);
    typename E::template Pix<XBLOCK> s;
    f.begin(s, x, y, iteration, phase);
    thread_window(f, s, windows + threadIdx.x, x, y);
    const int W = sv.W, H = sv.H;
    const long long base = sv.pix_off;
    const long long index = (long long)y * W + x;
    float4 b = d.hyp[base + index];
    float3 bn = make_float3(b.x, b.y, b.z);
    float bd = b.w;
    float best_cost = d.cost[base + index];
    for (int region = 0; region < 8; region++) {
        const int chosen = l3d_region_best(d.cost + base, region, x, y, W, H);
        if (chosen < 0) continue;
        float4 h = d.hyp[base + chosen];
        float3 hn = make_float3(h.x, h.y, h.z);
        float3 rq = f.ray_of((float)(chosen % W), (float)(chosen / W));
        float den = dot3f(hn, s.ray);
        if (fabsf(den) < 1e-6f) continue;
        float dd = dot3f(hn, make_float3(rq.x * h.w, rq.y * h.w, h.w)) / den;
        float c = f.cost_of(s, hn, dd);
        if (c < best_cost) {
            best_cost = c;
            bn = hn;
            bd = dd;
        }
    }
    float3 view = E::normalize(s.ray);
    float3 n_random = f.random_normal(s);
    float d_random = f.random_depth(s);
    float e = (fmaf(l3d_random(&s.rng), 2.0f, -1.0f) * 0.15f) * step;
    float d_perturbed = 1.0f / ((1.0f / bd) * (1.0f + e));
    float r1 = l3d_random(&s.rng), r2 = l3d_random(&s.rng), r3 = l3d_random(&s.rng);
    float3 n_perturbed = E::normalize(make_float3(bn.x + (fmaf(r1, 2.0f, -1.0f) * 0.6f) * step,
                                                    bn.y + (fmaf(r2, 2.0f, -1.0f) * 0.6f) * step,
                                                    bn.z + (fmaf(r3, 2.0f, -1.0f) * 0.6f) * step));
    if (dot3f(n_perturbed, view) >= 0.0f) n_perturbed = bn;
    const float3 cur_n = bn;
    const float cur_d = bd;
    for (int c = 0; c < 6; c++) {
        float3 nn = (c == 0 || c == 3) ? n_random : ((c == 1 || c == 5) ? n_perturbed : cur_n);
        float dv = (c == 0 || c == 2) ? d_random : ((c == 1 || c == 4) ? d_perturbed : cur_d);
        float cand = f.cost_of(s, nn, dv);
        if (cand < best_cost) {
            best_cost = cand;
            bn = nn;
            bd = dv;
        }
    }
    d.hyp[base + index] = make_float4(bn.x, bn.y, bn.z, bd);
    d.cost[base + index] = best_cost;
}

/* Blocks of 16 pixels, eight lanes each (l3d_lanes.cuh); a warp holds a 2 x 2 block of this
 * colour's pixels. */
constexpr int PARTS = TX * TY / 16;  /* blocks per tile of the propagate kernel */

template <class E>
__global__ void __launch_bounds__(128, E::kLayout.lane_blocks) k_fast_propagate_lanes(
        const L3dFastDev d, int iteration, int phase, float step) {
    __shared__ __align__(16) L3dFastView sv;
    __shared__ float2 windows[S * 16];
    const int tile = blockIdx.x / PARTS, part = blockIdx.x % PARTS;
    load_view(sv, d.views + find_view(d, tile));
    if (iteration >= sv.iterations) return;
    const int local = tile - sv.tile_start;
    const int warp = threadIdx.x >> 5, sub = (threadIdx.x >> 3) & 3, cand = threadIdx.x & 7;
    const int ty = (part >> 1) * 2 + (sub >> 1), tx = (part & 1) * (TX / 2) + warp * 2 + (sub & 1);
    int y = (local / sv.tiles_x) * TY + ty;
    int x = ((local % sv.tiles_x) * TX + tx) * 2 + ((y + phase) & 1);
    const bool inside = x < sv.W && y < sv.H;
    if (!__any_sync(0xffffffffu, inside)) return;
    x = min(x, sv.W - 1);  /* lanes outside the image stay for the shuffles and write nothing */
    y = min(y, sv.H - 1);
    E f(sv, d);
    typename E::template Pix<1> s;
    f.begin(s, x, y, iteration, phase);
    float2* win = windows + (warp * 4 + sub) * S;
    const float center = f.center(x, y);
    for (int i = cand; i < S; i += 8) win[i] = f.pair(x, y, i, center);
    __syncwarp();
    typename E::Sums sums;
#pragma unroll 6
    for (int i = 0; i < S; i++) sums.add(win[i]);
    f.finish(s, sums, center);
    __syncwarp();
    for (int i = cand; i < S; i += 8) win[i] = E::scale(win[i]);
    __syncwarp();
    s.win = win;
    l3d_step_lanes(f, s, d.hyp + sv.pix_off, d.cost + sv.pix_off, x, y, sv.W, sv.H, inside, cand, step);
}

__global__ void k_fast_pack(const L3dFastDev d) {
    const L3dFastView* v = d.views + blockIdx.y;
    if (!__ldg(&v->pack)) return;
    const int W = __ldg(&v->W), H = __ldg(&v->H);
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)W * H) return;
    const long long base = __ldg(&v->pix_off);
    float4 h = d.hyp[base + i];
    d.depths[__ldg(&v->ref_dep_off) + i] = pack_sample(h.w, make_float3(h.x, h.y, h.z), d.cost[base + i]);
}

template <class E>
__global__ void __launch_bounds__(128) k_fast_plane_cost(const L3dFastDev d, const float4* planes,
                                                         float* cost) {
    __shared__ __align__(16) L3dFastView sv;
    __shared__ float2 windows[S * XBLOCK];
    load_view(sv, d.views + find_view(d, blockIdx.x));
    const int local = blockIdx.x - sv.tile_start;
    const int y = (local / sv.tiles_x) * TY + threadIdx.x / TX;
    E f(sv, d);
    for (int half = 0; half < 2; half++) {
        const int x = (local % sv.tiles_x) * (2 * TX) + (threadIdx.x % TX) * 2 + half;
        if (x >= sv.W || y >= sv.H) continue;
        typename E::template Pix<XBLOCK> s;
        f.begin(s, x, y, 0, 0);
        thread_window(f, s, windows + threadIdx.x, x, y);
        const long long index = (long long)y * sv.W + x;
        float4 p = planes[sv.pix_off + index];
        cost[sv.pix_off + index] = f.cost_of(s, make_float3(p.x, p.y, p.z), p.w);
    }
}

}  // namespace

namespace {

template <class E>
cudaError_t launch_eval(int kernel, const L3dFastDev& d, int iteration, int phase, cudaStream_t st) {
    if (kernel == L3D_K_INIT) {
        k_fast_init<E><<<d.total_tiles, 128, 0, st>>>(d);
    } else {
        float step = ldexpf(1.0f, -iteration);
        const int sources = d.sources < 1 ? 1 : d.sources > 3 ? 3 : d.sources;
        if (d.total_tiles <= E::kLayout.lane_tiles[sources - 1])
            k_fast_propagate_lanes<E><<<d.total_tiles * PARTS, 128, 0, st>>>(d, iteration, phase, step);
        else
            k_fast_propagate<E><<<d.total_tiles, 128, 0, st>>>(d, iteration, phase, step);
    }
    return cudaGetLastError();
}

__global__ void k_make_pairs(const void* img, int storage, int W, int H, uint32_t* pairs) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const long long row = (long long)y * W;
    const int x1 = min(x + 1, W - 1);
    float a, b;
    if (storage == 0) {
        a = (float)((const uint8_t*)img)[row + x] / 255.0f;
        b = (float)((const uint8_t*)img)[row + x1] / 255.0f;
    } else if (storage == 1) {
        a = ((const float*)img)[row + x];
        b = ((const float*)img)[row + x1];
    } else if (storage == 2) {
        a = l3d_f16_to_f32(((const uint16_t*)img)[row + x]);
        b = l3d_f16_to_f32(((const uint16_t*)img)[row + x1]);
    } else {
        a = __uint_as_float((uint32_t)((const uint16_t*)img)[row + x] << 16);
        b = __uint_as_float((uint32_t)((const uint16_t*)img)[row + x1] << 16);
    }
    pairs[row + x] = l3d_f32_to_f16(a) | (l3d_f32_to_f16(b) << 16);
}

}  // namespace

cudaError_t l3d_launch_make_pairs(const void* img, int storage, int W, int H, uint32_t* pairs,
                                  cudaStream_t stream) {
    dim3 grid((W + 127) / 128, H);
    k_make_pairs<<<grid, 128, 0, stream>>>(img, storage, W, H, pairs);
    return cudaGetLastError();
}

/* variant = texture rows (6, 4, 3, 2; the exact evaluator, compensated sums and gathers take 6
 * only) + 16 x texture gathers with exact weights (fast evaluator, F16/F32/U8).  The quad (8) and
 * shared-window (32) bits of earlier kernels select nothing any more: both propagate kernels keep
 * the window in shared memory, and the thread-per-pixel one always maps quads to 2 x 2 pixels. */
cudaError_t l3d_launch_fast(int kernel, const L3dFastDev& d, int iteration, int phase, int variant,
                            cudaStream_t stream) {
    if (d.total_tiles <= 0) return cudaSuccess;
    if (kernel != L3D_K_INIT && kernel != L3D_K_PROPAGATE) return cudaErrorInvalidValue;
    const int rows = variant & 7;
    if (d.storage == 3 && !d.exact) { /* BF16 is sampled from linear memory */
        if (d.comp) return launch_eval<Fast<false, 6, true>>(kernel, d, iteration, phase, stream);
        return launch_eval<Fast<false, 6, false>>(kernel, d, iteration, phase, stream);
    }
    if (rows != 6 && (d.exact || d.comp || (variant & (16 | 32)) || !d.pairs)) return cudaErrorInvalidValue;
    if (d.exact) {
        if (d.comp) return launch_eval<Exact<true>>(kernel, d, iteration, phase, stream);
        return launch_eval<Exact<false>>(kernel, d, iteration, phase, stream);
    }
    if (variant & 16) { /* texture gathers with exact weights */
        if (d.comp) return launch_eval<Fast<true, 6, true, true>>(kernel, d, iteration, phase, stream);
        return launch_eval<Fast<true, 6, false, true>>(kernel, d, iteration, phase, stream);
    }
    if (d.comp) return launch_eval<Fast<true, 6, true>>(kernel, d, iteration, phase, stream);
    switch (rows) {
        case 6: return launch_eval<Fast<true, 6>>(kernel, d, iteration, phase, stream);
        case 4: return launch_eval<Fast<true, 4>>(kernel, d, iteration, phase, stream);
        case 3: return launch_eval<Fast<true, 3>>(kernel, d, iteration, phase, stream);
        case 2: return launch_eval<Fast<true, 2>>(kernel, d, iteration, phase, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t l3d_launch_fast_pack(const L3dFastDev& d, long long max_pixels, cudaStream_t stream) {
    if (d.n_views <= 0 || max_pixels <= 0) return cudaSuccess;
    dim3 grid((unsigned)((max_pixels + 255) / 256), (unsigned)d.n_views);
    k_fast_pack<<<grid, 256, 0, stream>>>(d);
    return cudaGetLastError();
}

cudaError_t l3d_launch_fast_plane_cost(const L3dFastDev& d, const float4* planes, float* cost,
                                       int variant, cudaStream_t stream) {
    if (d.total_tiles <= 0) return cudaSuccess;
    const int rows = variant & 7;
    const unsigned n = (unsigned)d.total_tiles;
    if (d.exact) {
        if (d.comp) k_fast_plane_cost<Exact<true>><<<n, 128, 0, stream>>>(d, planes, cost);
        else k_fast_plane_cost<Exact<false>><<<n, 128, 0, stream>>>(d, planes, cost);
    } else if (d.storage == 3) {
        if (d.comp) k_fast_plane_cost<Fast<false, 6, true>><<<n, 128, 0, stream>>>(d, planes, cost);
        else k_fast_plane_cost<Fast<false, 6>><<<n, 128, 0, stream>>>(d, planes, cost);
    } else if (variant & 16) {
        if (d.comp) k_fast_plane_cost<Fast<true, 6, true, true>><<<n, 128, 0, stream>>>(d, planes, cost);
        else k_fast_plane_cost<Fast<true, 6, false, true>><<<n, 128, 0, stream>>>(d, planes, cost);
    } else if (d.comp) {
        k_fast_plane_cost<Fast<true, 6, true>><<<n, 128, 0, stream>>>(d, planes, cost);
    } else if (rows == 6 || !d.pairs) {
        k_fast_plane_cost<Fast<true, 6>><<<n, 128, 0, stream>>>(d, planes, cost);
    } else if (rows == 4) {
        k_fast_plane_cost<Fast<true, 4>><<<n, 128, 0, stream>>>(d, planes, cost);
    } else if (rows == 3) {
        k_fast_plane_cost<Fast<true, 3>><<<n, 128, 0, stream>>>(d, planes, cost);
    } else {
        k_fast_plane_cost<Fast<true, 2>><<<n, 128, 0, stream>>>(d, planes, cost);
    }
    return cudaGetLastError();
}

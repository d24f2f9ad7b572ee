/* The range-restricted operations of csrc/l3d_ieee.h against the general ones; each kernel counts its
 * operands and the results that differ. */
#include <cuda_runtime.h>
#include <stdint.h>

#include "l3d_fmath.h"
#include "l3d_ieee.h"

namespace {

constexpr unsigned kBlocks = 148 * 8, kThreads = 256;

__device__ void tally(unsigned long long* counts, unsigned n, unsigned bad) {
    atomicAdd(counts, (unsigned long long)n);
    if (bad) atomicAdd(counts + 1, (unsigned long long)bad);
}

/* every float of the reciprocal's range */
__global__ void k_reciprocal(unsigned long long* counts) {
    unsigned n = 0, bad = 0;
    for (unsigned long long i = blockIdx.x * kThreads + threadIdx.x; i < 1ull << 32; i += kBlocks * kThreads) {
        const float x = __uint_as_float((uint32_t)i);
        if (!(fabsf(x) >= 0x1p-126f && fabsf(x) <= 0x1p125f)) continue;
        n++;
        if (__float_as_uint(l3d_rcp_normal(x)) != __float_as_uint(1.0f / x)) bad++;
    }
    tally(counts, n, bad);
}

/* Random quotients of the range, a third of them of whole numbers, a third with divisors of almost all-zero
 * or all-one mantissas, plain and with the divisor's reciprocal given.  A zero dividend's sign may be
 * lost. */
__global__ void k_quotient(unsigned long long* counts, uint32_t seed) {
    unsigned n = 0, bad = 0;
    uint32_t rng = l3d_pcg(seed ^ l3d_pcg(blockIdx.x * kThreads + threadIdx.x));
    for (int k = 0; k < 4096; k++) {
        uint32_t r[4];
        for (int j = 0; j < 4; j++) r[j] = rng = l3d_pcg(rng + 0x9e3779b9u);
        float a, b;
        if (r[2] % 3 == 0) {
            a = (float)(int)(r[0] >> (r[3] & 15)), b = (float)(1 + (r[1] >> (8 + (r[3] >> 4 & 15))));
        } else {
            uint32_t m = r[1] & 0x7fffffu;
            if (r[2] % 3 == 1) m = r[1] & 1 ? (r[1] >> 1 & 7u) : 0x7fffffu - (r[1] >> 1 & 7u);
            const int eb = 1 + (int)(r[2] >> 8 & 0xff) % 251;  /* 2^-126 .. 2^124 */
            const int ea = 27 + (int)(r[3] & 0xff) % 227;      /* 2^-100 .. 2^126 */
            b = __uint_as_float((r[2] & 0x80000000u) | (uint32_t)eb << 23 | m);
            a = __uint_as_float((r[3] & 0x80000000u) | (uint32_t)ea << 23 | (r[0] & 0x7fffffu));
        }
        const float q = a / b;
        if (a != 0.0f && !(fabsf(q) >= 0x1p-100f && fabsf(q) <= 0x1p100f)) continue;
        n++;
        const float p = l3d_div_normal(a, b), y = l3d_div_by(a, b, 1.0f / b);
        if (q == 0.0f ? !(p == 0.0f && y == 0.0f)
                      : __float_as_uint(p) != __float_as_uint(q) || __float_as_uint(y) != __float_as_uint(q))
            bad++;
    }
    tally(counts, n, bad);
}

/* every float as an index below n */
__global__ void k_index(unsigned long long* counts, unsigned n) {
    unsigned seen = 0, bad = 0;
    for (unsigned long long i = blockIdx.x * kThreads + threadIdx.x; i < 1ull << 32; i += kBlocks * kThreads) {
        const float x = __uint_as_float((uint32_t)i), r = rintf(x);
        const bool in = r >= 0.0f && r < (float)n;
        const unsigned at = l3d_rint_index(x);
        seen++;
        if (in != (at < n) || (in && at != (unsigned)r)) bad++;
    }
    tally(counts, seen, bad);
}

template <class F>
int count(F launch, unsigned long long* out) {
    unsigned long long* counts;
    cudaError_t e = cudaMalloc(&counts, 16);
    if (e != cudaSuccess) return (int)e;
    if ((e = cudaMemset(counts, 0, 16)) == cudaSuccess) {
        launch(counts);
        if ((e = cudaGetLastError()) == cudaSuccess) e = cudaMemcpy(out, counts, 16, cudaMemcpyDeviceToHost);
    }
    cudaFree(counts);
    return (int)e;
}

}  // namespace

extern "C" int check_reciprocal(unsigned long long* out) {
    return count([](unsigned long long* c) { k_reciprocal<<<kBlocks, kThreads>>>(c); }, out);
}
extern "C" int check_quotient(uint32_t seed, unsigned long long* out) {
    return count([=](unsigned long long* c) { k_quotient<<<kBlocks, kThreads>>>(c, seed); }, out);
}
extern "C" int check_index(uint32_t n, unsigned long long* out) {
    return count([=](unsigned long long* c) { k_index<<<kBlocks, kThreads>>>(c, n); }, out);
}

/*
 * Exclusive prefix sums of u32 or u64 counts on the device (stream compaction for surface extraction,
 * the brick lists, the brick grid and component removal).  Two launches: each block of 256 threads
 * sums a tile of 2048 elements, then scans its tile again behind the sum of the tiles before it, which
 * it adds up itself.  Above kFlat tiles a one-block launch between the two scans the tiles' sums, so
 * that the blocks need not each read them all.  Deterministic: the result does not depend on
 * scheduling.  In-place (out == in) works: a block reads its tile before it writes it.
 *
 * A scan's cost here is its launches, not its bytes: the brick counts of 384^3 (110592) took five
 * launches of 2.1 to 2.9 us each when a level scanned 1024 elements and added its sums back.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "l3d_internal.h"

namespace {

constexpr int kThreads = 256;
constexpr int kPer = 8;
constexpr int kTile = kThreads * kPer;
constexpr long long kFlat = 1024;  /* tiles whose sums every block adds up itself */

template <typename T>
__device__ __forceinline__ T warp_inclusive(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const T t = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += t;
    }
    return v;
}

/* Sum of one value per thread, in every thread. */
template <typename T>
__device__ __forceinline__ T block_sum(T v) {
    __shared__ T part[kThreads / 32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    T s = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; i++) s += part[i];
    return s;
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_scan_sums(const T* in, long long n, T* sums) {
    const long long base = (long long)blockIdx.x * kTile + threadIdx.x;
    T v = 0;
#pragma unroll
    for (int i = 0; i < kPer; i++) {
        const long long j = base + (long long)i * kThreads;
        if (j < n) v += in[j];
    }
    v = block_sum(v);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
}

/* One block: exclusive scan of the tiles' sums, kTile at a time.  Each step is a chain of loads, a scan and
 * two barriers, so its length counts: with one sum per thread and step, building a grid of 400^3 cells took
 * 677 us and of 1000^3 9.35 ms, with kPer 633 us and 8.63 ms. */
template <typename T>
__global__ void __launch_bounds__(kThreads) k_scan_top(T* sums, long long tiles) {
    __shared__ T warps[kThreads / 32];
    T carry = 0;
    for (long long at = 0; at < tiles; at += kTile) {
        const long long base = at + (long long)threadIdx.x * kPer;
        T v[kPer];
        T local = 0;
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            v[i] = base + i < tiles ? sums[base + i] : 0;
            local += v[i];
        }
        const T inc = warp_inclusive(local);
        if ((threadIdx.x & 31) == 31) warps[threadIdx.x >> 5] = inc;
        __syncthreads();
        T run = carry + inc - local, all = 0;
#pragma unroll
        for (int i = 0; i < kThreads / 32; i++) {
            if (i < (int)(threadIdx.x >> 5)) run += warps[i];
            all += warps[i];
        }
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            if (base + i < tiles) sums[base + i] = run;
            run += v[i];
        }
        carry += all;
        __syncthreads();
    }
}

/* flat: sums[] are the tiles' sums; otherwise their exclusive scan. */
template <typename T>
__global__ void __launch_bounds__(kThreads) k_scan_apply(const T* in, T* out, long long n, const T* sums, bool flat,
                                                         T* total) {
    __shared__ T warps[kThreads / 32];
    const long long base = (long long)blockIdx.x * kTile + (long long)threadIdx.x * kPer;
    T v[kPer];
    T local = 0;
#pragma unroll
    for (int i = 0; i < kPer; i++) {
        v[i] = base + i < n ? in[base + i] : 0;
        local += v[i];
    }
    T before = 0;
    if (flat) {
        T p = 0;
        for (unsigned j = threadIdx.x; j < blockIdx.x; j += kThreads) p += sums[j];
        before = block_sum(p);
    } else {
        before = sums[blockIdx.x];
    }
    const T inc = warp_inclusive(local);
    if ((threadIdx.x & 31) == 31) warps[threadIdx.x >> 5] = inc;
    __syncthreads();
    for (int i = 0; i < (int)(threadIdx.x >> 5); i++) before += warps[i];
    T run = before + inc - local;
#pragma unroll
    for (int i = 0; i < kPer; i++) {
        if (base + i < n) out[base + i] = run;
        run += v[i];
    }
    /* the thread that holds the last element has the sum of all */
    if (total && base < n && base + kPer >= n) *total = run;
}

long long tiles_of(long long n) { return (n + kTile - 1) / kTile; }

template <typename T>
cudaError_t scan(const T* in, T* out, long long n, T* sums, T* total, cudaStream_t stream) {
    if (n <= 0) {
        if (total) return cudaMemsetAsync(total, 0, sizeof(T), stream);
        return cudaSuccess;
    }
    const long long tiles = tiles_of(n);
    const bool flat = tiles <= kFlat;
    k_scan_sums<T><<<(unsigned)tiles, kThreads, 0, stream>>>(in, n, sums);
    if (!flat) k_scan_top<T><<<1, kThreads, 0, stream>>>(sums, tiles);
    k_scan_apply<T><<<(unsigned)tiles, kThreads, 0, stream>>>(in, out, n, sums, flat, total);
    return cudaGetLastError();
}

}  // namespace

size_t l3d_scan_scratch(long long n) { return (size_t)(tiles_of(n) + 1) * sizeof(uint32_t); }
size_t l3d_scan64_scratch(long long n) { return (size_t)(tiles_of(n) + 1) * sizeof(unsigned long long); }

int l3d_scan_launches(long long n) { return n <= 0 ? 0 : (tiles_of(n) <= kFlat ? 2 : 3); }

cudaError_t l3d_scan_exclusive(const uint32_t* in, uint32_t* out, long long n, uint32_t* scratch,
                               uint32_t* total, cudaStream_t stream) {
    return scan<uint32_t>(in, out, n, scratch, total, stream);
}

cudaError_t l3d_scan64_exclusive(const unsigned long long* in, unsigned long long* out, long long n,
                                 unsigned long long* scratch, unsigned long long* total, cudaStream_t stream) {
    return scan<unsigned long long>(in, out, n, scratch, total, stream);
}

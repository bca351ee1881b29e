// Multi-block inclusive scan (reduce, scan of the tile sums, apply) of 32- and
// 64-bit values, used by the planning of the ion lists.
//
// A warp takes 512 (64-bit: 256) neighbouring values in four 16-byte accesses
// per lane, so every access of the apply pass is coalesced: bound by HBM.
// (Sixteen consecutive values per thread, four bytes an access, reached 1.2
// TB/s: 35 us for the 5.6 M coverage counters of the 20,000-protein database.)
#pragma once
#include <cstdint>
#include "device_common.cuh"

namespace hfx {

constexpr int kScanThreads = 256, kScanSteps = 4;
template <typename T> constexpr int kScanVec = 16 / (int)sizeof(T);                       // values per access
template <typename T> constexpr int kScanWarp = 32 * kScanVec<T> * kScanSteps;            // values per warp
template <typename T> constexpr int kScanTile = kScanWarp<T> * (kScanThreads / 32);       // values per block

template <typename T>
__device__ __forceinline__ T warp_scan_of(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T t = __shfl_up_sync(kFullMask, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

__device__ __forceinline__ bool on_16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// The warp's values of one tile, as 16-byte vectors where they lie on 16-byte
// boundaries (zero beyond n).
template <typename T>
__device__ __forceinline__ void scan_load(const T *a, int64_t n, int64_t at, T (&v)[kScanSteps][kScanVec<T>]) {
    const int lane = threadIdx.x & 31;
    const bool wide = on_16(a);
#pragma unroll
    for (int k = 0; k < kScanSteps; ++k) {
        const int64_t i = at + (int64_t)(k * 32 + lane) * kScanVec<T>;
        if (wide && i + kScanVec<T> <= n) {
            const uint4 u = *reinterpret_cast<const uint4 *>(a + i);
            const T *w = reinterpret_cast<const T *>(&u);
#pragma unroll
            for (int j = 0; j < kScanVec<T>; ++j) v[k][j] = w[j];
        } else {
#pragma unroll
            for (int j = 0; j < kScanVec<T>; ++j) v[k][j] = i + j < n ? a[i + j] : T(0);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const T *__restrict__ a, int64_t n, T *__restrict__ partial) {
    __shared__ T red[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T v[kScanSteps][kScanVec<T>];
    scan_load(a, n, (int64_t)blockIdx.x * kScanTile<T> + (int64_t)warp * kScanWarp<T>, v);
    T s = 0;
#pragma unroll
    for (int k = 0; k < kScanSteps; ++k)
#pragma unroll
        for (int j = 0; j < kScanVec<T>; ++j) s += v[k][j];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(kFullMask, s, o);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kScanThreads / 32; ++w) s += red[w];
        partial[blockIdx.x] = s;
    }
}

// Exclusive scan of the tile sums in place, one block.
template <typename T>
__global__ void __launch_bounds__(1024) k_scan_partials(T *__restrict__ partial, int64_t nb) {
    __shared__ T ws[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T carry = 0;
    for (int64_t b0 = 0; b0 < nb; b0 += 1024) {
        const int64_t i = b0 + threadIdx.x;
        const T v = i < nb ? partial[i] : T(0);
        const T x = warp_scan_of(v);
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        if (warp == 0) ws[lane] = warp_scan_of(ws[lane]);
        __syncthreads();
        if (i < nb) partial[i] = carry + (warp ? ws[warp - 1] : T(0)) + x - v;
        carry += ws[31];
        __syncthreads();
    }
}

// Inclusive scan of one tile from its block's offset: out[i] = sum a[0..i];
// out may be a.
template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const T *a, int64_t n, const T *__restrict__ partial,
                                                             T *out) {
    __shared__ T ws[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = (int64_t)blockIdx.x * kScanTile<T> + (int64_t)warp * kScanWarp<T>;
    T v[kScanSteps][kScanVec<T>];
    scan_load(a, n, at, v);
    T carry = 0;
#pragma unroll
    for (int k = 0; k < kScanSteps; ++k) {
#pragma unroll
        for (int j = 1; j < kScanVec<T>; ++j) v[k][j] += v[k][j - 1];
        const T own = v[k][kScanVec<T> - 1], x = warp_scan_of(own);
#pragma unroll
        for (int j = 0; j < kScanVec<T>; ++j) v[k][j] += carry + x - own;
        carry += __shfl_sync(kFullMask, x, 31);
    }
    if (lane == 0) ws[warp] = carry;
    __syncthreads();
    T before = partial[blockIdx.x];
    for (int w = 0; w < warp; ++w) before += ws[w];
    const bool wide = on_16(out);
#pragma unroll
    for (int k = 0; k < kScanSteps; ++k) {
        const int64_t i = at + (int64_t)(k * 32 + lane) * kScanVec<T>;
#pragma unroll
        for (int j = 0; j < kScanVec<T>; ++j) v[k][j] += before;
        if (wide && i + kScanVec<T> <= n) {
            uint4 u;
            T *w = reinterpret_cast<T *>(&u);
#pragma unroll
            for (int j = 0; j < kScanVec<T>; ++j) w[j] = v[k][j];
            *reinterpret_cast<uint4 *>(out + i) = u;
        } else {
#pragma unroll
            for (int j = 0; j < kScanVec<T>; ++j)
                if (i + j < n) out[i + j] = v[k][j];
        }
    }
}

// partial holds scan_partials(n).
template <typename T>
inline int64_t scan_partials(int64_t n) { return (n + kScanTile<T> - 1) / kScanTile<T> + 1; }
template <typename T>
inline int scan_inclusive(const T *in, int64_t n, T *out, T *partial, cudaStream_t st) {
    if (n <= 0) return 0;
    const int64_t nb = (n + kScanTile<T> - 1) / kScanTile<T>;
    k_scan_reduce<T><<<(unsigned)nb, kScanThreads, 0, st>>>(in, n, partial);
    k_scan_partials<T><<<1, 1024, 0, st>>>(partial, nb);
    k_scan_apply<T><<<(unsigned)nb, kScanThreads, 0, st>>>(in, n, partial, out);
    return (int)cudaGetLastError();
}

}  // namespace hfx

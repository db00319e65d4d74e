// Exclusive prefix sums of int64 values given by a functor of the index (so
// counts, flags and widths need no pass of their own).  Up to kScanOne values
// take one CTA and one launch; more take a launch of tiles, whose local sums
// land in out and whose totals in tmp, and one that adds every tile's offset.
#pragma once

#include "common.cuh"

namespace sdb {
namespace scan {

constexpr int kItems = 8, kThreads = 256, kTile = kThreads * kItems;
constexpr int kOneThreads = 1024, kOne = kOneThreads * kItems;  // one CTA's step; kScanOne values in one launch
constexpr size_t kScanOne = kOne;
constexpr int kSumsInSmem = 1024;  // tiles whose totals a consumer scans by itself

// Exclusive sum of v over the block's THREADS threads; the block's total.
template <int THREADS> __device__ __forceinline__ int64_t block_exclusive(int64_t v, int64_t* total) {
    __shared__ int64_t wsum[THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int64_t o = __shfl_up_sync(0xffffffffu, x, s);
        if (lane >= s) x += o;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int64_t y = lane < THREADS / 32 ? wsum[lane] : 0;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const int64_t o = __shfl_up_sync(0xffffffffu, y, s);
            if (lane >= s) y += o;
        }
        if (lane < THREADS / 32) wsum[lane] = y;
    }
    __syncthreads();
    const int64_t before = w ? wsum[w - 1] : 0;
    *total = wsum[THREADS / 32 - 1];
    __syncthreads();
    return before + x - v;
}

template <int THREADS, class In>
__device__ __forceinline__ int64_t scan_step(const In& in, int64_t* out, size_t base0, size_t n, int64_t carry) {
    const size_t base = base0 + (size_t)threadIdx.x * kItems;
    int64_t v[kItems], s = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        v[i] = base + i < n ? in(base + i) : 0;
        s += v[i];
    }
    int64_t total;
    int64_t ex = carry + block_exclusive<THREADS>(s, &total);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (base + i < n) out[base + i] = ex;
        ex += v[i];
    }
    return total;
}

template <class In> __global__ void __launch_bounds__(kOneThreads) k_scan_one(In in, int64_t* out, size_t n) {
    scan_step<kOneThreads>(in, out, 0, n, 0);
}

template <class In>
__global__ void __launch_bounds__(kThreads) k_scan_tiles(In in, int64_t* out, size_t n, int64_t* sums) {
    const int64_t total = scan_step<kThreads>(in, out, (size_t)blockIdx.x * kTile, n, 0);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// scanned: sums hold the tiles' offsets already.
static __global__ void __launch_bounds__(kThreads) k_scan_finish(int64_t* out, size_t n, const int64_t* sums,
                                                                 int scanned) {
    int64_t off = 0;
    if (scanned) {
        off = sums[blockIdx.x];
    } else {
        int64_t s = 0;
        for (int t = threadIdx.x; t < (int)blockIdx.x; t += kThreads) s += sums[t];
        block_exclusive<kThreads>(s, &off);
    }
    const size_t end = min(n, (size_t)(blockIdx.x + 1) * kTile);
    for (size_t j = (size_t)blockIdx.x * kTile + threadIdx.x; j < end; j += kThreads) out[j] += off;
}

struct Load64 {
    const int64_t* p;
    __device__ int64_t operator()(size_t i) const { return p[i]; }
};
// n values and zeros behind them
struct Load32 {
    const int32_t* p;
    size_t n;
    __device__ int64_t operator()(size_t i) const { return i < n ? p[i] : 0; }
};

inline size_t tiles(size_t n) { return (n + kTile - 1) / kTile; }

// The tiles only: local sums in out, totals in tmp (tiles(n) of them); one
// launch.  For consumers that add the offsets themselves.
template <class In> int launch_local(const In& in, int64_t* out, size_t n, int64_t* tmp, cudaStream_t st) {
    k_scan_tiles<<<(unsigned)tiles(n), kThreads, 0, st>>>(in, out, n, tmp);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <class In> int launch(const In& in, int64_t* out, size_t n, int64_t* tmp, cudaStream_t st) {
    if (n == 0) return 0;
    if (n <= kScanOne) {
        k_scan_one<<<1, kOneThreads, 0, st>>>(in, out, n);
        return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
    }
    const size_t nb = tiles(n);
    if (launch_local(in, out, n, tmp, st) < 0) return -1;
    int launches = 2;
    if (nb > 4096) {  // beyond this, every tile adding up the ones before it costs more than a scan of them
        const int r = launch(Load64{tmp}, tmp, nb, tmp + nb + 1, st);
        if (r < 0) return -1;
        launches += r;
    }
    k_scan_finish<<<(unsigned)nb, kThreads, 0, st>>>(out, n, tmp, nb > 4096 ? 1 : 0);
    return cudaPeekAtLastError() == cudaSuccess ? launches : -1;
}

}  // namespace scan
}  // namespace sdb

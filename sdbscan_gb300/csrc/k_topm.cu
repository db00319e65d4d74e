// Stage 2: per random vector, the m largest ("close") and m smallest ("far")
// projections over all points — matrix_topM of rp_parIndex
// (src/sDbscan.cpp:151-208).
//
// Exact without a per-vector heap over n:
//  1. The projection kernel leaves, for every chunk of points, the maximum
//     and minimum projection onto each vector (as BF16 rounded away from the
//     extreme, so still bounds of attained values; 32-bit keys where the caller made them).  The m-th largest of the chunk
//     maxima is a value attained by m different points, so it is a lower
//     bound T on the true m-th largest value (k_thresholds).
//  2. One pass over the projections appends every (value, point) with value
//     >= T to the vector's candidate list (k_collect).  All of the top m are
//     in it.
//  3. An exact sort of each candidate list by (value desc, point asc) yields
//     the top m (k_select).  A list whose candidates overflow its buffer is
//     resolved by an exact radix select over the whole column (select_column).
// Ties: the reference's heap keeps, among equal values at the boundary, the
// ones its heap order dictates; this engine keeps the smallest point ids and
// counts such boundary ties.
#include "common.cuh"

#include <algorithm>

namespace sdb {
namespace {

// Block-wide bitonic sort (descending) of `len` (power of two) u64 keys in smem.
__device__ void block_sort_desc(uint64_t* s, int len) {
    for (int size = 2; size <= len; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int i = threadIdx.x; i < len / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (stride - 1));
                const int hi = lo + stride;
                const bool desc = (lo & size) == 0;
                const uint64_t a = s[lo], b = s[hi];
                if ((a < b) == desc) {
                    s[lo] = b;
                    s[hi] = a;
                }
            }
        }
    }
    __syncthreads();
}

__host__ __device__ inline int pow2_ceil(int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

// T of every list (r, side): the m-th largest chunk extreme, 0 with fewer than
// m of them.  A CTA takes `cols` neighbouring vectors (32-byte row segments with
// 8), folds `group` chunks into one (their maximum is attained too) and keeps
// the results' order-preserving keys in shared memory; a warp then finds a list's
// m-th largest key by bisection, counting once per bit of a key.
// The chunks folded into one are ng apart, each layer of ng rotated against the
// one before: points that arrive cluster after cluster, or in several such
// runs, keep about as many chunks of their own as without folding.  (Folding
// neighbours leaves a cluster of n / 40 points fewer than m = 50 of them, the
// bound drops to the next cluster and every list overflows: top-m stage of 1M x
// 64 in 40 clusters 0.91 ms shuffled, 68 sorted by cluster.)
// A 32-bit radix select with a histogram per list, and one CTA per column of
// two float arrays, read 8 times the bytes, sent every key of a list (one
// binade) at the same few bins and had one thread walk them: 104 us at any n
// above 44K, D = 1024 (45 at 2K); this takes 30 (14), about half of it the
// bisections.
constexpr int kThrThreads = 512;
// A chunk's extremes (TopMArgs::chunkExt, chunkKeys) as the keys of both sides.
struct Keys16 {
    static constexpr int kBits = 16;
    typedef uint32_t Pair;  // close side in the low half
    static __device__ __forceinline__ Pair none() { return 0xffffffffu; }  // as loaded: the least keys
    static __device__ __forceinline__ Pair load(const TopMArgs& a, size_t at) { return __ldg(a.chunkExt + at); }
    static __device__ __forceinline__ Pair keys(Pair b) {  // a set sign bit flips its half, else that bit alone flips
        return b ^ (((b >> 15) & 0x00010001u) * 0x7fffu | 0x80008000u);
    }
    static __device__ __forceinline__ Pair larger(Pair x, Pair y) {
        Pair z;
        asm("max.u16x2 %0, %1, %2;" : "=r"(z) : "r"(x), "r"(y));
        return z;
    }
    static __device__ __forceinline__ uint32_t of(Pair x, int side) { return side ? x >> 16 : x & 0xffffu; }
};
struct Keys32 {
    static constexpr int kBits = 32;
    typedef uint2 Pair;
    static __device__ __forceinline__ Pair none() { return make_uint2(0u, 0u); }
    static __device__ __forceinline__ Pair load(const TopMArgs& a, size_t at) { return __ldg(a.chunkKeys + at); }
    static __device__ __forceinline__ Pair keys(Pair b) { return b; }
    static __device__ __forceinline__ Pair larger(Pair x, Pair y) { return make_uint2(max(x.x, y.x), max(x.y, y.y)); }
    static __device__ __forceinline__ uint32_t of(Pair x, int side) { return side ? x.y : x.x; }
};

template <class K>
__global__ void __launch_bounds__(kThrThreads) k_thresholds(TopMArgs a, int cols, int group, int ng) {
    extern __shared__ __align__(8) unsigned char thrShm[];
    typename K::Pair* keys = reinterpret_cast<typename K::Pair*>(thrShm);  // ng x stride
    const int stride = cols | 1;
    const int c = threadIdx.x & (cols - 1), r = blockIdx.x * cols + c, step = kThrThreads / cols;
    if (r < a.nproj) {
        const int turn = ng / 8 * 5;
        for (int q = threadIdx.x / cols; q < ng; q += step) {
            typename K::Pair most = K::keys(K::none());
            int x = q;
            for (int j = 0; j < group; j += 8) {  // eight loads in flight
                typename K::Pair e[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int g = (j + u) * ng + x;
                    e[u] = g < a.G ? K::load(a, (size_t)g * a.nproj + r) : K::none();
                    x += turn;
                    if (x >= ng) x -= ng;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) most = K::larger(most, K::keys(e[u]));
            }
            keys[q * stride + c] = most;
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int l = threadIdx.x >> 5; l < 2 * cols; l += kThrThreads / 32) {
        const int col = l >> 1, side = l & 1, rr = blockIdx.x * cols + col;
        if (rr >= a.nproj) break;
        uint32_t t = 0;
        if (ng >= a.m) {
            for (int bit = K::kBits - 1; bit >= 0; --bit) {
                const uint32_t at = t | (1u << bit);
                int cnt = 0;
#pragma unroll 8
                for (int q = lane; q < ng; q += 32) cnt += K::of(keys[q * stride + col], side) >= at;
                if (warp_sum(cnt) >= a.m) t = at;
            }
            t <<= 32 - K::kBits;  // the smallest 32-bit key with these high bits
        }
        if (lane == 0) (side ? a.thrMin : a.thrMax)[rr] = __uint_as_float(t);  // raw key bits
    }
}

// A block takes kCollectRows consecutive points; a thread takes 4
// consecutive vectors of them (16-byte loads, all rows' loads issued before
// any compare, the vectors' thresholds loaded once).
constexpr int kCollectRows = 8;
__global__ void __launch_bounds__(256) k_collect(TopMArgs a) {
    const int per_row = a.nproj / 4;
    const int p0 = blockIdx.x * kCollectRows;
    for (int c4 = threadIdx.x; c4 < per_row; c4 += blockDim.x) {
        const int r0 = c4 * 4;
        float4 v4[kCollectRows];
#pragma unroll
        for (int i = 0; i < kCollectRows; ++i)
            v4[i] = p0 + i < a.n ? __ldcs(reinterpret_cast<const float4*>(a.P + (size_t)(p0 + i) * a.nproj) + c4)
                                 : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float4 tcv = __ldg(reinterpret_cast<const float4*>(a.thrMax) + c4);
        const float4 tfv = __ldg(reinterpret_cast<const float4*>(a.thrMin) + c4);
        const uint32_t tc[4] = {__float_as_uint(tcv.x), __float_as_uint(tcv.y), __float_as_uint(tcv.z),
                                __float_as_uint(tcv.w)};
        const uint32_t tf[4] = {__float_as_uint(tfv.x), __float_as_uint(tfv.y), __float_as_uint(tfv.z),
                                __float_as_uint(tfv.w)};
#pragma unroll
        for (int i = 0; i < kCollectRows; ++i) {
            const int p = p0 + i;
            if (p >= a.n) break;
            const float vv[4] = {v4[i].x, v4[i].y, v4[i].z, v4[i].w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int r = r0 + t;
                const uint32_t kc = key_of(vv[t]);
                const uint32_t kf = key_of(-vv[t]);
                if (kc >= tc[t]) {
                    const int slot = atomicAdd(a.candCount + r, 1);
                    if (slot < a.cap)
                        a.cand[(size_t)r * a.cap + slot] = ((uint64_t)kc << 32) | (uint32_t)(0xffffffffu - (uint32_t)p);
                }
                if (kf >= tf[t]) {
                    const int list = a.nproj + r;
                    const int slot = atomicAdd(a.candCount + list, 1);
                    if (slot < a.cap)
                        a.cand[(size_t)list * a.cap + slot] =
                            ((uint64_t)kf << 32) | (uint32_t)(0xffffffffu - (uint32_t)p);
                }
            }
        }
    }
}

// The same where a thread expects a pass of its own (n <= kDenseCollect topM):
// the passing rows of each vector and side are found first and their places
// taken by one atomicAdd, so the eight round trips overlap instead of one
// following the other (2K points, where one value in twenty passes: 25 us
// serially, 11 here; 50K, one in a thousand: 57 and 75).
constexpr int kDenseCollect = 128;
__global__ void __launch_bounds__(256) k_collect_dense(TopMArgs a) {
    const int per_row = a.nproj / 4;
    const int p0 = blockIdx.x * kCollectRows;
    const int rows = min(kCollectRows, a.n - p0);
    for (int c4 = threadIdx.x; c4 < per_row; c4 += blockDim.x) {
        const int r0 = c4 * 4;
        float4 v4[kCollectRows];
#pragma unroll
        for (int i = 0; i < kCollectRows; ++i)
            v4[i] = i < rows ? __ldcs(reinterpret_cast<const float4*>(a.P + (size_t)(p0 + i) * a.nproj) + c4)
                             : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float4 tcv = __ldg(reinterpret_cast<const float4*>(a.thrMax) + c4);
        const float4 tfv = __ldg(reinterpret_cast<const float4*>(a.thrMin) + c4);
        const uint32_t tc[4] = {__float_as_uint(tcv.x), __float_as_uint(tcv.y), __float_as_uint(tcv.z),
                                __float_as_uint(tcv.w)};
        const uint32_t tf[4] = {__float_as_uint(tfv.x), __float_as_uint(tfv.y), __float_as_uint(tfv.z),
                                __float_as_uint(tfv.w)};
        uint32_t pass[8];  // per vector, close and far side: the passing rows
        uint32_t any = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            pass[2 * t] = pass[2 * t + 1] = 0;
#pragma unroll
            for (int i = 0; i < kCollectRows; ++i) {
                const float v = t == 0 ? v4[i].x : t == 1 ? v4[i].y : t == 2 ? v4[i].z : v4[i].w;
                if (key_of(v) >= tc[t]) pass[2 * t] |= 1u << i;
                if (key_of(-v) >= tf[t]) pass[2 * t + 1] |= 1u << i;
            }
            pass[2 * t] &= (1u << rows) - 1u;
            pass[2 * t + 1] &= (1u << rows) - 1u;
            any |= pass[2 * t] | pass[2 * t + 1];
        }
        if (!any) continue;
        int slot[8];
#pragma unroll
        for (int s = 0; s < 8; ++s)
            slot[s] = pass[s] ? atomicAdd(a.candCount + (s & 1) * a.nproj + r0 + s / 2, __popc(pass[s])) : 0;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const size_t list = (size_t)((s & 1) * a.nproj + r0 + s / 2);
#pragma unroll
            for (int i = 0; i < kCollectRows; ++i) {
                if (!((pass[s] >> i) & 1u)) continue;
                const float v = s / 2 == 0 ? v4[i].x : s / 2 == 1 ? v4[i].y : s / 2 == 2 ? v4[i].z : v4[i].w;
                if (slot[s] < a.cap)
                    a.cand[list * a.cap + slot[s]] =
                        ((uint64_t)key_of(s & 1 ? -v : v) << 32) | (uint32_t)(0xffffffffu - (uint32_t)(p0 + i));
                ++slot[s];
            }
        }
    }
}

// Generic (nproj % 4 != 0) variant: one thread per projection.
__global__ void k_collect1(TopMArgs a) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)a.n * a.nproj;
    if (q >= total) return;
    const int p = (int)(q / a.nproj);
    const int r = (int)(q % a.nproj);
    const float v = a.P[q];
    const uint32_t kc = key_of(v), kf = key_of(-v);
    if (kc >= __float_as_uint(a.thrMax[r])) {
        const int slot = atomicAdd(a.candCount + r, 1);
        if (slot < a.cap) a.cand[(size_t)r * a.cap + slot] = ((uint64_t)kc << 32) | (uint32_t)(0xffffffffu - (uint32_t)p);
    }
    if (kf >= __float_as_uint(a.thrMin[r])) {
        const int list = a.nproj + r;
        const int slot = atomicAdd(a.candCount + list, 1);
        if (slot < a.cap) a.cand[(size_t)list * a.cap + slot] = ((uint64_t)kf << 32) | (uint32_t)(0xffffffffu - (uint32_t)p);
    }
}

// Exact radix select over a whole column, for lists whose candidate buffer
// overflowed (heavy ties, adversarial orderings).  sk: shared memory, m entries
// rounded up to a power of two.
__device__ void select_column(const TopMArgs& a, int list, uint64_t* sk) {
    __shared__ uint32_t hist[256];
    __shared__ uint32_t prefix, prefixMask;
    __shared__ int need;  // how many of the remaining (prefix-matching) elements we still take
    __shared__ int above; // elements strictly above the final key
    __shared__ int taken;
    const int r = list % a.nproj, side = list / a.nproj;
    auto keyAt = [&](int p) -> uint32_t {
        const float v = a.P[(size_t)p * a.nproj + r];
        return side == 0 ? key_of(v) : key_of(-v);
    };
    if (threadIdx.x == 0) {
        prefix = 0;
        prefixMask = 0;
        need = a.m;
        above = 0;
    }
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        for (int p = threadIdx.x; p < a.n; p += blockDim.x) {
            const uint32_t k = keyAt(p);
            if ((k & prefixMask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int acc = 0;
            for (int b = 255; b >= 0; --b) {
                if (acc + (int)hist[b] >= need) {
                    prefix |= (uint32_t)b << shift;
                    prefixMask |= 255u << shift;
                    above += acc;
                    need -= acc;
                    break;
                }
                acc += hist[b];
            }
        }
        __syncthreads();
    }
    // prefix is now the exact m-th largest key K; `above` elements are > K and
    // `need` elements equal to K are taken, smallest point ids first.
    const uint32_t K = prefix;
    const int len = pow2_ceil(max(a.m, 2));
    for (int i = threadIdx.x; i < len; i += blockDim.x) sk[i] = 0;
    if (threadIdx.x == 0) taken = 0;
    __syncthreads();
    __shared__ int eqTaken;
    if (threadIdx.x == 0) eqTaken = 0;
    __syncthreads();
    // strictly greater: any order
    for (int p = threadIdx.x; p < a.n; p += blockDim.x) {
        const uint32_t k = keyAt(p);
        if (k > K) {
            const int s = atomicAdd(&taken, 1);
            sk[s] = ((uint64_t)k << 32) | (uint32_t)(0xffffffffu - (uint32_t)p);
        }
    }
    __syncthreads();
    // equal: in ascending point order, block-sequential chunks
    int eqTotal = 0;
    for (int base = 0; base < a.n; base += blockDim.x) {
        const int p = base + threadIdx.x;
        const bool eq = p < a.n && keyAt(p) == K;
        const int cnt = __syncthreads_count(eq);
        // rank within the chunk
        const unsigned bal = __ballot_sync(0xffffffffu, eq);
        __shared__ int warpCnt[32];
        const int w = threadIdx.x >> 5;
        if ((threadIdx.x & 31) == 0) warpCnt[w] = __popc(bal);
        __syncthreads();
        int before = 0;
        for (int ww = 0; ww < w; ++ww) before += warpCnt[ww];
        before += __popc(bal & ((1u << (threadIdx.x & 31)) - 1u));
        const int rank = eqTaken + before;
        if (eq && rank < need) sk[above + rank] = ((uint64_t)K << 32) | (uint32_t)(0xffffffffu - (uint32_t)p);
        __syncthreads();
        if (threadIdx.x == 0) eqTaken += cnt;
        eqTotal += cnt;
        __syncthreads();
    }
    block_sort_desc(sk, len);
    for (int i = threadIdx.x; i < a.m; i += blockDim.x)
        a.topM[(size_t)r * 2 * a.m + side * a.m + i] = (int32_t)(0xffffffffu - (uint32_t)sk[i]);
    if (threadIdx.x == 0 && eqTotal > need) atomicAdd(a.ties, 1ull);
}

// One CTA per list: exact sort of the candidates, first m written to topM.
__global__ void k_select(TopMArgs a) {
    extern __shared__ uint64_t sk[];
    const int list = blockIdx.x;
    const int r = list % a.nproj, side = list / a.nproj;
    const int c = a.candCount[list];
    if (c > a.cap) {
        select_column(a, list, sk);
        return;
    }
    const int len = pow2_ceil(max(c, 2));
    for (int i = threadIdx.x; i < len; i += blockDim.x) sk[i] = i < c ? a.cand[(size_t)list * a.cap + i] : 0ull;
    block_sort_desc(sk, len);
    // c >= m always holds (the threshold is attained by >= m points); if it
    // ever did not, point 0 stands in and the fit reports an internal error.
    for (int i = threadIdx.x; i < a.m; i += blockDim.x)
        a.topM[(size_t)r * 2 * a.m + side * a.m + i] = i < c ? (int32_t)(0xffffffffu - (uint32_t)sk[i]) : 0;
    if (threadIdx.x == 0 && c < a.m) atomicExch(a.errFlag, 1);
    if (threadIdx.x == 0 && c > a.m && (sk[a.m - 1] >> 32) == (sk[a.m] >> 32)) atomicAdd(a.ties, 1ull);
}

}  // namespace

template <class K> static int launch_thresholds(const TopMArgs& a, cudaStream_t st) {
    // 912 groups or 4m: enough that the m-th largest is close to the m-th value
    const int group = std::max(1, a.G / std::max(912, 4 * a.m));
    const int ng = (a.G + group - 1) / group;
    int cols = 8;
    while (cols > 1 && sizeof(typename K::Pair) * (size_t)ng * (cols | 1) > 100 * 1024) cols >>= 1;
    const size_t sm = sizeof(typename K::Pair) * (size_t)ng * (cols | 1);
    if (sm > 48 * 1024 &&
        cudaFuncSetAttribute(k_thresholds<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
        return -1;
    k_thresholds<K><<<(a.nproj + cols - 1) / cols, kThrThreads, sm, st>>>(a, cols, group, ng);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_topm_thresholds(const TopMArgs& a, cudaStream_t st) {
    return a.chunkKeys != nullptr ? launch_thresholds<Keys32>(a, st) : launch_thresholds<Keys16>(a, st);
}

int launch_topm_collect(const TopMArgs& a, cudaStream_t st) {
    if (a.nproj % 4 == 0 && (reinterpret_cast<uintptr_t>(a.P) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(a.thrMax) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.thrMin) & 15) == 0) {
        const int threads = std::min(256, (a.nproj / 4 + 31) / 32 * 32);
        const unsigned blocks = (unsigned)((a.n + kCollectRows - 1) / kCollectRows);
        if (a.n <= (int64_t)kDenseCollect * a.m) k_collect_dense<<<blocks, threads, 0, st>>>(a);
        else k_collect<<<blocks, threads, 0, st>>>(a);
    } else {
        const size_t total = (size_t)a.n * a.nproj;
        k_collect1<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a);
    }
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_topm_select(const TopMArgs& a, cudaStream_t st) {
    const size_t sm = sizeof(uint64_t) * pow2_ceil(a.cap);
    if (sm > 48 * 1024 &&
        cudaFuncSetAttribute(k_select, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
        return -1;
    k_select<<<2 * a.nproj, 256, sm, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace sdb

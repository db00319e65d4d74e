// sngDbscan / sngOptics neighbourhoods on the packed distance tile
// (pair_block.cuh), for the distances that have one (all but JS): the block of
// one shared sample (k_sng.cu has the rule and the scalar form) and the
// samples per 32 points (k_sng_blocks.cu).  The columns -- the sampled points,
// or a block's own 32 points -- come from a dimension-major copy, the rows
// from the transformed data.
// Against the scalar tiles: 200K x 784 with 1990 sampled points 14.2 -> 11.3 ms,
// 50K x 784 with 500 draws a point 0.99 -> 0.87 (copy included).
#include "pair_block.cuh"
#include "sng_draws.cuh"

#include <climits>

namespace sdb {
namespace {

using namespace ptile;

// Column j of tile t: the point at t CT + j of ids (null: that point itself).
struct ArrayCols {
    const int32_t* ids;
    int count, CT;
    __device__ int operator()(int64_t t, int j) const {
        const int64_t c = t * CT + j;
        return c < count ? (ids != nullptr ? __ldg(ids + c) : (int)c) : -1;
    }
};

struct NoVisit {
    __device__ void operator()(int, int, int, float, float, bool, bool) const {}
};

// 128 consecutive points x 64 sampled ones; tiles of a row block are
// consecutive so that a wave shares its rows in L2.
struct BlockSmem {
    PairSmem<Shape64> t;
    int colW[Shape64::CT];
    int passTotal;
};

template <int DIST>
__global__ void __launch_bounds__(kThreads, 3) k_sng_pair(SngArgs a) {
    using S = Shape64;
    extern __shared__ __align__(16) unsigned char raw[];
    BlockSmem& sm = *reinterpret_cast<BlockSmem*>(raw);
    const int tid = threadIdx.x;
    const int rb = (int)(blockIdx.x / a.nct), ct = (int)(blockIdx.x % a.nct);
    const int p0 = rb * S::TM, rows = min(S::TM, a.n - p0);
    const ArrayCols cols{a.cols, a.nU, S::CT};
    for (int i = tid; i < S::TM; i += kThreads) sm.t.rowLoad[i] = p0 + (i < rows ? i : 0);
    for (int j = tid; j < S::CT; j += kThreads) {
        const int q = cols(ct, j);
        sm.t.colPoint[j] = q;
        sm.colW[j] = q >= 0 && a.mult != nullptr ? __ldg(a.mult + ct * S::CT + j) : 1;
    }
    if (tid == 0) sm.passTotal = 0;
    pair_tile<DIST, S>(PairTile{a.Xt, a.ld, a.eps, a.colCopy + (size_t)ct * a.ld * S::CTP, rows}, sm.t, a.small,
                       NoVisit{});
    int pass = 0;
    for (int row = tid; row < rows; row += kThreads) {
        const u64 w = ((u64)sm.t.mask[2 * row + 1] << 32) | sm.t.mask[2 * row];
        if (a.mask != nullptr) a.mask[(size_t)ct * a.n + p0 + row] = w;
        pass += __popcll(w);
        if (!w) continue;
        int s = 0;
        for (u64 b = w; b; b &= b - 1) s += sm.colW[__ffsll((long long)b) - 1];
        atomicAdd(a.rowDeg + p0 + row, s);
    }
    for (int j = tid; j < S::CT; j += kThreads)
        if (sm.t.colCount[j]) atomicAdd(a.colCnt + ct * S::CT + j, sm.t.colCount[j]);
    pass = warp_sum(pass);
    if ((tid & 31) == 0 && pass) atomicAdd(&sm.passTotal, pass);
    __syncthreads();
    if (tid == 0 && sm.passTotal) atomicAdd(a.pairs, (unsigned long long)sm.passTotal);
}

// sngOptics: the tile's distances, 32 floats per draw, for k_sngb_insert.
struct StoreDraws {
    float* dists;  // of the tile's first draw
    __device__ void operator()(int row, int, int c, float d0, float d1, bool, bool) const {
        *reinterpret_cast<float2*>(dists + (size_t)row * kSngBlockRows + c) = make_float2(d0, d1);
    }
};

// 192 draws of a 32-point block x its points.
template <int DIST, bool STORE>
__global__ void __launch_bounds__(kThreads, 3) k_sngb_pair(SngBlockArgs a) {
    using S = Shape32;
    static_assert(S::CT == kSngBlockRows, "a block's points are the tile's columns");
    extern __shared__ __align__(16) unsigned char raw[];
    struct Smem {
        PairSmem<S> t;
        int passTotal;
    };
    Smem& sm = *reinterpret_cast<Smem*>(raw);
    const int tid = threadIdx.x;
    const int64_t nT = (a.S + S::TM - 1) / S::TM;
    const int64_t b = (int64_t)blockIdx.x / nT, j0 = (int64_t)blockIdx.x % nT * S::TM;
    const int rows = (int)min((int64_t)S::TM, a.S - j0);
    for (int i = tid; i < S::TM; i += kThreads)
        sm.t.rowLoad[i] = block_draw(a.key, a.S, b, j0 + (i < rows ? i : 0), a.n);
    const ArrayCols cols{nullptr, a.n, S::CT};
    for (int j = tid; j < S::CT; j += kThreads) sm.t.colPoint[j] = cols(b, j);
    if (tid == 0) sm.passTotal = 0;
    const PairTile tile{a.Xt, a.ld, a.eps, a.colCopy + (size_t)b * a.ld * S::CTP, rows};
    if constexpr (STORE)
        pair_tile<DIST, S>(tile, sm.t, a.small, StoreDraws{a.dists + (size_t)(b * a.S + j0) * kSngBlockRows});
    else
        pair_tile<DIST, S>(tile, sm.t, a.small, NoVisit{});
    int pass = 0;
    for (int row = tid; row < rows; row += kThreads) {
        const uint32_t w = sm.t.mask[2 * row];
        a.words[b * a.S + j0 + row] = w;
        pass += __popc(w);
        if (w) atomicAdd(a.degree + sm.t.rowLoad[row], __popc(w));  // the draw's side
    }
    if (tid < S::CT && sm.t.colCount[tid]) atomicAdd(a.degree + sm.t.colPoint[tid], sm.t.colCount[tid]);
    pass = warp_sum(pass);
    if ((tid & 31) == 0 && pass) atomicAdd(&sm.passTotal, pass);
    __syncthreads();
    if (tid == 0 && sm.passTotal) atomicAdd(a.pairs, (unsigned long long)sm.passTotal);
}

// sngOptics: every passing pair into both points' tables, a thread per (block,
// draw) word, from the stored distances.  (Computing the tiles a second time
// to insert from their registers: 1727 us at 50K x 784, p = 0.01, against
// 167 here.)
__global__ void __launch_bounds__(256) k_sngb_insert(SngBlockArgs a) {
    const int64_t total = (int64_t)((a.n + kSngBlockRows - 1) / kSngBlockRows) * a.S;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    uint32_t w = __ldg(a.words + i);
    if (!w) return;
    const int64_t b = i / a.S;
    const int q = block_draw(a.key, a.S, b, i % a.S, a.n);
    for (; w; w &= w - 1) {
        const int c = __ffs((int)w) - 1;
        const float d = __ldg(a.dists + (size_t)i * kSngBlockRows + c);
        hash_insert(a, (int)b * kSngBlockRows + c, q, d);
        hash_insert(a, q, (int)b * kSngBlockRows + c, d);
    }
}

template <class K> bool room(K kernel, size_t sm) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) == cudaSuccess;
}

template <int DIST> int launch_block_d(const SngArgs& a, cudaStream_t st) {
    const int64_t tiles = (int64_t)((a.n + Shape64::TM - 1) / Shape64::TM) * a.nct;
    if (tiles > INT_MAX || !room(k_sng_pair<DIST>, sizeof(BlockSmem))) return -1;
    k_sng_pair<DIST><<<(unsigned)tiles, kThreads, sizeof(BlockSmem), st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <int DIST, bool STORE> int launch_sngb_d(const SngBlockArgs& a, cudaStream_t st) {
    const int64_t nT = (a.S + Shape32::TM - 1) / Shape32::TM;
    const int64_t tiles = (int64_t)((a.n + kSngBlockRows - 1) / kSngBlockRows) * nT;
    const size_t sm = sizeof(PairSmem<Shape32>) + 16;
    if (tiles <= 0) return 0;
    if (tiles > INT_MAX || !room(k_sngb_pair<DIST, STORE>, sm)) return -1;
    k_sngb_pair<DIST, STORE><<<(unsigned)tiles, kThreads, sm, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <int DIST> int launch_sngb_s(const SngBlockArgs& a, cudaStream_t st) {
    return a.dists != nullptr ? launch_sngb_d<DIST, true>(a, st) : launch_sngb_d<DIST, false>(a, st);
}

}  // namespace

size_t sng_pair_bytes(int dist, int64_t cols, int ld) {
    return dist == DIST_JS ? 0 : sizeof(float) * (size_t)((cols + 63) / 64 * 64) * ld;
}

int launch_sng_cols(const SngArgs& a, cudaStream_t st) {
    return launch_col_tiles(a.Xt, a.ld, a.dist, ArrayCols{a.cols, a.nU, Shape64::CT}, a.nct, Shape64::CT, Shape64::CTP,
                            a.colCopy, st);
}

int launch_sng_pair(const SngArgs& a, cudaStream_t st) {
    if (a.n <= 0 || a.nct <= 0) return 0;
    switch (a.dist) {
        case DIST_COSINE: return launch_block_d<DIST_COSINE>(a, st);
        case DIST_L1: return launch_block_d<DIST_L1>(a, st);
        case DIST_L2: return launch_block_d<DIST_L2>(a, st);
        case DIST_CHI2: return launch_block_d<DIST_CHI2>(a, st);
    }
    return -1;
}

int launch_sngb_cols(const SngBlockArgs& a, cudaStream_t st) {
    return launch_col_tiles(a.Xt, a.ld, a.dist, ArrayCols{nullptr, a.n, Shape32::CT},
                            (a.n + kSngBlockRows - 1) / kSngBlockRows, Shape32::CT, Shape32::CTP, a.colCopy, st);
}

int launch_sngb_pair(const SngBlockArgs& a, cudaStream_t st) {
    switch (a.dist) {
        case DIST_COSINE: return launch_sngb_s<DIST_COSINE>(a, st);
        case DIST_L1: return launch_sngb_s<DIST_L1>(a, st);
        case DIST_L2: return launch_sngb_s<DIST_L2>(a, st);
        case DIST_CHI2: return launch_sngb_s<DIST_CHI2>(a, st);
    }
    return -1;
}

int launch_sngb_insert(const SngBlockArgs& a, cudaStream_t st) {
    const int64_t total = (int64_t)((a.n + kSngBlockRows - 1) / kSngBlockRows) * a.S;
    if (total <= 0) return 0;
    k_sngb_insert<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace sdb

// A CTA's work around the packed distance tile (pair_tile.cuh), shared by the
// candidate distances (k_dist_pair.cu) and the sampled neighbourhoods of
// sngDbscan / sngOptics (k_sng_pair.cu): the dimension-major column copies,
// the tile's shared memory, its pass bits and counts.
//
// A tile is rarely full at the end of a list or a sample (50K points, k = 5, D
// = 1024: 244 members a list), so it runs with 2, 4, 6 or 8 rows per thread,
// whatever holds its rows: the work follows the rows to a quarter of a tile.
#pragma once

#include "pair_tile.cuh"

namespace sdb {
namespace ptile {

// The rows of a column tile, dimension-major: tile t holds ld runs of CTP
// floats, run k the k-th dimension of its CT columns' points (zero where cols
// gives no point); negated but for Cosine.  cols(t, j): the point of column j.
constexpr int kCtDims = 128;
template <class Cols>
__global__ void __launch_bounds__(256) k_col_tiles(const float* __restrict__ Xt, int ld, Cols cols, int CT, int CTP,
                                                   int negate, float* __restrict__ outAll) {
    __shared__ float tile[64][kCtDims + 1];
    const int64_t t = blockIdx.x;
    const int k0 = blockIdx.y * kCtDims, kn = min(kCtDims, ld - k0);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = w; j < CTP; j += 8) {
        const int p = j < CT ? cols(t, j) : -1;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (p >= 0 && 4 * lane < kn) {
            v = __ldg(reinterpret_cast<const float4*>(Xt + (size_t)p * ld + k0) + lane);
            if (negate) v = make_float4(-v.x, -v.y, -v.z, -v.w);
        }
        tile[j][4 * lane] = v.x;
        tile[j][4 * lane + 1] = v.y;
        tile[j][4 * lane + 2] = v.z;
        tile[j][4 * lane + 3] = v.w;
    }
    __syncthreads();
    const int q4 = CTP / 4;
    float4* out = reinterpret_cast<float4*>(outAll + ((size_t)t * ld + k0) * CTP);
    for (int e = threadIdx.x; e < kn * q4; e += blockDim.x) {
        const int k = e / q4, q = e % q4;
        out[e] = make_float4(tile[4 * q][k], tile[4 * q + 1][k], tile[4 * q + 2][k], tile[4 * q + 3][k]);
    }
}

template <class Cols>
int launch_col_tiles(const float* Xt, int ld, int dist, const Cols& cols, int64_t tiles, int CT, int CTP, float* out,
                     cudaStream_t st) {
    if (tiles <= 0) return 0;
    const dim3 grid((unsigned)tiles, (unsigned)((ld + kCtDims - 1) / kCtDims));
    k_col_tiles<<<grid, 256, 0, st>>>(Xt, ld, cols, CT, CTP, dist == DIST_COSINE ? 0 : 1, out);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <class S> struct PairSmem {
    float As[NST * S::TM * LDA];
    float Bs[NST * KT * S::CTP];
    int rowLoad[S::TM];   // the rows' points (past the tile's rows, its first one: staged, not used)
    int colPoint[S::CT];  // -1: no column
    int colCount[S::CT];  // passes per column out
    unsigned mask[2 * S::TM];  // pass bits per row out (bit j: column j)
};

// What a tile is computed from: the rows' data, eps, its column copy.
struct PairTile {
    const float* Xt;
    int ld;
    float eps;
    const float* cols;
    int rows;
};

// Distances of a tile with up to RG * RM rows, its pass bits (dist <= eps, not
// the point itself) and column counts.  visit(row, p, c, d0, d1, pass0, pass1)
// for every row's column pairs c, c + 1, also those without a column.
template <int DIST, class S, int RM, class Visit>
__device__ __forceinline__ void pair_rows(const PairTile& a, PairSmem<S>& sm, Visit& visit) {
    constexpr int kFinish = DIST == DIST_CHI2_ANY ? DIST_CHI2 : DIST;
    u64 acc[RM][S::CN / 2];
    pair_accumulate<DIST, S, RM>(a.Xt, a.ld, sm.rowLoad, a.cols, sm.As, sm.Bs, acc);
    if (!S::active(threadIdx.x)) return;
    int rg, tx;
    S::coords(threadIdx.x, rg, tx);
    int colPass[S::CN];
#pragma unroll
    for (int j = 0; j < S::CN; ++j) colPass[j] = 0;
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int row = rg + S::RG * i;
        if (row >= a.rows) continue;
        const int p = sm.rowLoad[row];
        u64 bits = 0;
#pragma unroll
        for (int j = 0; j < S::CN / 2; ++j) {
            const int c = S::column(tx, j);
            float d0, d1;
            unpack2(acc[i][j], d0, d1);
            d0 = dtile::finish<kFinish>(d0);
            d1 = dtile::finish<kFinish>(d1);
            const int q0 = sm.colPoint[c], q1 = sm.colPoint[c + 1];
            const bool p0 = d0 <= a.eps && q0 >= 0 && q0 != p, p1 = d1 <= a.eps && q1 >= 0 && q1 != p;
            colPass[2 * j] += p0;
            colPass[2 * j + 1] += p1;
            bits |= (u64)((p0 ? 1u : 0u) | (p1 ? 2u : 0u)) << c;
            visit(row, p, c, d0, d1, p0, p1);
        }
        if ((unsigned)bits) atomicOr(&sm.mask[2 * row], (unsigned)bits);
        if ((unsigned)(bits >> 32)) atomicOr(&sm.mask[2 * row + 1], (unsigned)(bits >> 32));
    }
#pragma unroll
    for (int j = 0; j < S::CN; ++j)
        if (colPass[j]) atomicAdd(&sm.colCount[S::column(tx, j >> 1) + (j & 1)], colPass[j]);
}

// The whole tile: rowLoad and colPoint filled by the caller (not synchronised
// yet), mask and colCount complete on return (synchronised).  small: Chi2
// flags per point (DistArgs::small).
template <int DIST, class S, class Visit>
__device__ __forceinline__ void pair_tile(const PairTile& a, PairSmem<S>& sm, const uint8_t* small, Visit visit) {
    const int tid = threadIdx.x;
    for (int i = tid; i < 2 * S::TM; i += kThreads) sm.mask[i] = 0;
    for (int j = tid; j < S::CT; j += kThreads) sm.colCount[j] = 0;
    __syncthreads();
    bool any = false;  // Chi2: a row or a column of the tile has an entry below kChi2Small
    if (DIST == DIST_CHI2) {
        for (int i = tid; i < a.rows; i += kThreads) any |= small[sm.rowLoad[i]] != 0;
        for (int j = tid; j < S::CT; j += kThreads) any |= sm.colPoint[j] >= 0 && small[sm.colPoint[j]] != 0;
        any = __syncthreads_or(any);
    }
    const int need = (a.rows + S::RG - 1) / S::RG;  // rows per thread
    if (DIST == DIST_CHI2 && any) pair_rows<DIST_CHI2_ANY, S, S::RMAX>(a, sm, visit);
    else if (need <= 2) pair_rows<DIST, S, 2>(a, sm, visit);
    else if (need <= 4) pair_rows<DIST, S, 4>(a, sm, visit);
    else if (S::RMAX == 6 || need <= 6) pair_rows<DIST, S, 6>(a, sm, visit);
    else pair_rows<DIST, S, S::RMAX>(a, sm, visit);
    __syncthreads();
}

using Shape32 = PairShape<4, 8, 6>;
using Shape40 = PairShape<5, 8, 8>;
using Shape50 = PairShape<5, 10, 8>;
using Shape64 = PairShape<8, 8, 8>;

}  // namespace ptile
}  // namespace sdb

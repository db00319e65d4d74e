// Stage 4, the packed tile: candidate distances and the eps test of
// rp_findCorePoints / rp_findCoreDist (src/sDbscan.cpp:243-359, :1323-1412)
// for Cosine, L1, L2 and Chi2 with the packed FP32 tile of pair_tile.cuh.
//
// Tile = (list l, TM member rows, CT candidate columns), as in k_dist.cu; the
// candidate rows come from a dimension-major copy that k_cand_tiles writes
// once per fit (0.13 ms at 1M x 784, D = 1024, m = 50: every list's tile is
// then one contiguous run per stage, read by about 50 row tiles).
//
// A list's last tile is rarely full (50K points, k = 5, D = 1024: 244 members
// a list), so a tile runs with 2, 4, 6 or 8 rows per thread, whatever holds
// its rows: the work follows the members to 48 rows instead of 192.
//
// Bound: the FP32 FMA pipe (72 % active at 1M x 784).
#include "pair_tile.cuh"

#include <algorithm>
#include <climits>

namespace sdb {
namespace {

using namespace ptile;

// The lists' candidate rows, dimension-major: column tile t = l nct + ct holds
// ld runs of CTP floats, run k the k-th dimension of its CT candidates (zero
// for columns past m); negated for L1 / L2.
constexpr int kCtDims = 128;
__global__ void __launch_bounds__(256) k_cand_tiles(DistArgs a, int CTP, int negate) {
    __shared__ float tile[64][kCtDims + 1];
    const int l = blockIdx.x / a.nct, ct = blockIdx.x % a.nct;
    const int r = l % a.nproj, side = l / a.nproj;
    const int32_t* cand = a.topM + (size_t)r * 2 * a.m + side * a.m;
    const int k0 = blockIdx.y * kCtDims, kn = min(kCtDims, a.ld - k0);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = w; j < CTP; j += 8) {
        const int c = ct * a.CT + j;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (j < a.CT && c < a.m && 4 * lane < kn) {
            v = __ldg(reinterpret_cast<const float4*>(a.Xt + (size_t)__ldg(cand + c) * a.ld + k0) + lane);
            if (negate) v = make_float4(-v.x, -v.y, -v.z, -v.w);
        }
        tile[j][4 * lane] = v.x;
        tile[j][4 * lane + 1] = v.y;
        tile[j][4 * lane + 2] = v.z;
        tile[j][4 * lane + 3] = v.w;
    }
    __syncthreads();
    const int q4 = CTP / 4;
    float4* out = reinterpret_cast<float4*>(a.cand + ((size_t)blockIdx.x * a.ld + k0) * CTP);
    for (int e = threadIdx.x; e < kn * q4; e += blockDim.x) {
        const int k = e / q4, q = e % q4;
        out[e] = make_float4(tile[4 * q][k], tile[4 * q + 1][k], tile[4 * q + 2][k], tile[4 * q + 3][k]);
    }
}

template <class S> struct PairSmem {
    float As[NST * S::TM * LDA];
    float Bs[NST * KT * S::CTP];
    int rowLoad[S::TM];   // point whose row is staged (the first member's past the tile's rows)
    int rowSlot[S::TM];
    int colPoint[S::CT];  // -1 past m
    int colCount[S::CT];
    unsigned mask[2 * S::TM];
    int passTotal;
};

// Distances of a tile with up to RG * RM rows, and its pass bits, column
// counts and (optionally) distances.
template <int DIST, class S, int RM>
__device__ __forceinline__ void pair_rows(const DistArgs& a, PairSmem<S>& sm, int rows, const float* cand, int ct) {
    constexpr int kFinish = DIST == DIST_CHI2_ANY ? DIST_CHI2 : DIST;
    u64 acc[RM][S::CN / 2];
    pair_accumulate<DIST, S, RM>(a.Xt, a.ld, sm.rowLoad, cand, sm.As, sm.Bs, acc);
    if (!S::active(threadIdx.x)) return;
    int rg, tx;
    S::coords(threadIdx.x, rg, tx);
    int colPass[S::CN];
#pragma unroll
    for (int j = 0; j < S::CN; ++j) colPass[j] = 0;
    const int left = a.m - ct * S::CT;  // columns of this tile
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int row = rg + S::RG * i;
        if (row >= rows) continue;
        const int p = sm.rowLoad[row];
        float* dist = a.dists == nullptr ? nullptr
                                         : a.dists + ((size_t)p * 2 * a.k + sm.rowSlot[row]) * a.m + ct * S::CT;
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
            if (dist != nullptr) {
                if (c < left) dist[c] = d0;
                if (c + 1 < left) dist[c + 1] = d1;
            }
        }
        if ((unsigned)bits) atomicOr(&sm.mask[2 * row], (unsigned)bits);
        if ((unsigned)(bits >> 32)) atomicOr(&sm.mask[2 * row + 1], (unsigned)(bits >> 32));
    }
#pragma unroll
    for (int j = 0; j < S::CN; ++j)
        if (colPass[j]) atomicAdd(&sm.colCount[S::column(tx, j >> 1) + (j & 1)], colPass[j]);
}

template <int DIST, class S>
__global__ void __launch_bounds__(kThreads, 3) k_dist_pair(DistArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    PairSmem<S>& sm = *reinterpret_cast<PairSmem<S>*>(raw);
    const int tid = threadIdx.x;
    if ((int64_t)blockIdx.x >= *a.tileTotal) return;
    const int64_t t = tile_at(a.tilePerm, blockIdx.x);
    const int l = a.tileList[t];
    const int64_t ti = t - a.tileOff[l];
    const int mt = (int)(ti / a.nct), ct = (int)(ti % a.nct);
    const int64_t mbeg = a.listOff[l] + (int64_t)mt * S::TM;
    const int rows = (int)min((int64_t)S::TM, a.listOff[l + 1] - mbeg);
    const int r = l % a.nproj, side = l / a.nproj;
    const int32_t* list = a.topM + (size_t)r * 2 * a.m + side * a.m;
    for (int i = tid; i < S::TM; i += kThreads) {
        const int2 mb = a.members[mbeg + (i < rows ? i : 0)];
        sm.rowLoad[i] = mb.x;
        sm.rowSlot[i] = mb.y;
        sm.mask[2 * i] = 0;
        sm.mask[2 * i + 1] = 0;
    }
    for (int j = tid; j < S::CT; j += kThreads) {
        const int c = ct * S::CT + j;
        sm.colPoint[j] = c < a.m ? list[c] : -1;
        sm.colCount[j] = 0;
    }
    if (tid == 0) sm.passTotal = 0;
    bool small = false;  // Chi2: a row or a candidate of the tile has an entry below kChi2Small
    if (DIST == DIST_CHI2) {
        for (int i = tid; i < rows; i += kThreads) small |= a.small[sm.rowLoad[i]] != 0;
        for (int j = tid; j < S::CT; j += kThreads) small |= sm.colPoint[j] >= 0 && a.small[sm.colPoint[j]] != 0;
    }
    small = __syncthreads_or(small);

    const float* cand = a.cand + ((size_t)l * a.nct + ct) * a.ld * S::CTP;
    const int need = (rows + S::RG - 1) / S::RG;  // rows per thread
    if (DIST == DIST_CHI2 && small) pair_rows<DIST_CHI2_ANY, S, S::RMAX>(a, sm, rows, cand, ct);
    else if (need <= 2) pair_rows<DIST, S, 2>(a, sm, rows, cand, ct);
    else if (need <= 4) pair_rows<DIST, S, 4>(a, sm, rows, cand, ct);
    else if (S::RMAX == 6 || need <= 6) pair_rows<DIST, S, 6>(a, sm, rows, cand, ct);
    else pair_rows<DIST, S, S::RMAX>(a, sm, rows, cand, ct);
    __syncthreads();

    int pass = 0;
    for (int row = tid; row < rows; row += kThreads) {
        const u64 w = ((u64)sm.mask[2 * row + 1] << 32) | sm.mask[2 * row];
        a.masks[((size_t)sm.rowLoad[row] * 2 * a.k + sm.rowSlot[row]) * a.W + ct] = w;
        pass += __popcll(w);
    }
    for (int j = tid; j < S::CT; j += kThreads)
        if (sm.colCount[j]) atomicAdd(a.inRaw + sm.colPoint[j], sm.colCount[j]);
    pass = warp_sum(pass);
    if ((tid & 31) == 0 && pass) atomicAdd(&sm.passTotal, pass);
    __syncthreads();
    if (tid == 0 && sm.passTotal) atomicAdd(a.pairs, (unsigned long long)sm.passTotal);
}

using Shape32 = PairShape<4, 8, 6>;
using Shape40 = PairShape<5, 8, 8>;
using Shape50 = PairShape<5, 10, 8>;
using Shape64 = PairShape<8, 8, 8>;

template <int DIST, class S> int launch_pair_t(const DistArgs& a, cudaStream_t st) {
    const size_t sm = sizeof(PairSmem<S>);
    if (cudaFuncSetAttribute(k_dist_pair<DIST, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) !=
        cudaSuccess)
        return -1;
    k_dist_pair<DIST, S><<<(unsigned)a.nTiles, kThreads, sm, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <int DIST> int launch_pair_d(const DistArgs& a, cudaStream_t st) {
    switch (a.CT) {
        case 32: return launch_pair_t<DIST, Shape32>(a, st);
        case 40: return launch_pair_t<DIST, Shape40>(a, st);
        case 50: return launch_pair_t<DIST, Shape50>(a, st);
        case 64: return launch_pair_t<DIST, Shape64>(a, st);
    }
    return -1;
}

}  // namespace

// The columns per tile whose tiles take the least time for m candidates: the
// cost of one column tile of each shape, in columns of the 64-wide one.
int pair_tile_cols(int dist, int m) {
    if (dist != DIST_COSINE && dist != DIST_L1 && dist != DIST_L2 && dist != DIST_CHI2) return 0;
    static const int shape[4][2] = {{64, 640}, {50, 542}, {40, 450}, {32, 370}};
    int best = 0, cols = 0;
    for (const auto& s : shape) {
        const int cost = (m + s[0] - 1) / s[0] * s[1];
        if (cols == 0 || cost < best) {
            best = cost;
            cols = s[0];
        }
    }
    return cols;
}

int pair_tile_rows(int cols) {
    return cols == 32 ? Shape32::TM : cols == 40 ? Shape40::TM : cols == 50 ? Shape50::TM : Shape64::TM;
}

static int pair_tile_ctp(int cols) { return (cols + 3) / 4 * 4; }

size_t pair_cand_bytes(int cols, int nproj, int m, int ld) {
    return sizeof(float) * (size_t)2 * nproj * ((m + cols - 1) / cols) * ld * pair_tile_ctp(cols);
}

int launch_cand_tiles(const DistArgs& a, cudaStream_t st) {
    const dim3 grid((unsigned)(2 * a.nproj * a.nct), (unsigned)((a.ld + kCtDims - 1) / kCtDims));
    k_cand_tiles<<<grid, 256, 0, st>>>(a, pair_tile_ctp(a.CT), a.dist == DIST_COSINE ? 0 : 1);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_dist_pair(const DistArgs& a, cudaStream_t st) {
    if (a.nTiles <= 0) return 0;
    if (a.nTiles > INT_MAX) return -1;
    switch (a.dist) {
        case DIST_COSINE: return launch_pair_d<DIST_COSINE>(a, st);
        case DIST_L1: return launch_pair_d<DIST_L1>(a, st);
        case DIST_L2: return launch_pair_d<DIST_L2>(a, st);
        case DIST_CHI2: return launch_pair_d<DIST_CHI2>(a, st);
    }
    return -1;
}

}  // namespace sdb

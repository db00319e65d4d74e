// Stage 4, the packed tile: candidate distances and the eps test of
// rp_findCorePoints / rp_findCoreDist (src/sDbscan.cpp:243-359, :1323-1412)
// for Cosine, L1, L2 and Chi2 with the packed FP32 tile of pair_tile.cuh.
//
// Tile = (list l, TM member rows, CT candidate columns), as in k_dist.cu; the
// candidate rows come from a dimension-major copy that k_col_tiles writes
// once per fit (0.13 ms at 1M x 784, D = 1024, m = 50: every list's tile is
// then one contiguous run per stage, read by about 50 row tiles).
//
// Bound: the FP32 FMA pipe (72 % active at 1M x 784).
#include "pair_block.cuh"

#include <algorithm>
#include <climits>

namespace sdb {
namespace {

using namespace ptile;

// The columns of list tile t = l nct + ct.
struct ListCols {
    const int32_t* topM;
    int nproj, m, nct, CT;
    __device__ int operator()(int64_t t, int j) const {
        const int l = (int)(t / nct), c = (int)(t % nct) * CT + j;
        return c < m ? __ldg(topM + (size_t)(l % nproj) * 2 * m + (l / nproj) * m + c) : -1;
    }
};

// Writes the distances of a tile's pairs (sOPTICS and sweeps).
template <class S, bool STORE> struct StoreDists {
    const DistArgs& a;
    const int* rowSlot;
    int ct;
    __device__ void operator()(int row, int p, int c, float d0, float d1, bool, bool) const {
        if (!STORE) return;
        const int left = a.m - ct * S::CT;  // columns of this tile
        float* d = a.dists + ((size_t)p * 2 * a.k + rowSlot[row]) * a.m + ct * S::CT;
        if (c < left) d[c] = d0;
        if (c + 1 < left) d[c + 1] = d1;
    }
};

template <class S> struct DistSmem {
    PairSmem<S> t;
    int rowSlot[S::TM];
    int passTotal;
};

template <int DIST, class S, bool STORE>
__global__ void __launch_bounds__(kThreads, 3) k_dist_pair(DistArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    DistSmem<S>& sm = *reinterpret_cast<DistSmem<S>*>(raw);
    const int tid = threadIdx.x;
    if ((int64_t)blockIdx.x >= *a.tileTotal) return;
    const int64_t t = tile_at(a.tilePerm, blockIdx.x);
    const int l = a.tileList[t];
    const int64_t ti = t - a.tileOff[l];
    const int mt = (int)(ti / a.nct), ct = (int)(ti % a.nct);
    const int64_t mbeg = a.listOff[l] + (int64_t)mt * S::TM;
    const int rows = (int)min((int64_t)S::TM, a.listOff[l + 1] - mbeg);
    const ListCols cols{a.topM, a.nproj, a.m, a.nct, S::CT};
    for (int i = tid; i < S::TM; i += kThreads) {
        const int2 mb = a.members[mbeg + (i < rows ? i : 0)];
        sm.t.rowLoad[i] = mb.x;
        sm.rowSlot[i] = mb.y;
    }
    for (int j = tid; j < S::CT; j += kThreads) sm.t.colPoint[j] = cols((int64_t)l * a.nct + ct, j);
    if (tid == 0) sm.passTotal = 0;
    pair_tile<DIST, S>(PairTile{a.Xt, a.ld, a.eps, a.cand + ((size_t)l * a.nct + ct) * a.ld * S::CTP, rows}, sm.t,
                       a.small, StoreDists<S, STORE>{a, sm.rowSlot, ct});

    int pass = 0;
    for (int row = tid; row < rows; row += kThreads) {
        const u64 w = ((u64)sm.t.mask[2 * row + 1] << 32) | sm.t.mask[2 * row];
        a.masks[((size_t)sm.t.rowLoad[row] * 2 * a.k + sm.rowSlot[row]) * a.W + ct] = w;
        pass += __popcll(w);
    }
    for (int j = tid; j < S::CT; j += kThreads)
        if (sm.t.colCount[j]) atomicAdd(a.inRaw + sm.t.colPoint[j], sm.t.colCount[j]);
    pass = warp_sum(pass);
    if ((tid & 31) == 0 && pass) atomicAdd(&sm.passTotal, pass);
    __syncthreads();
    if (tid == 0 && sm.passTotal) atomicAdd(a.pairs, (unsigned long long)sm.passTotal);
}

template <int DIST, class S, bool STORE> int launch_pair_s(const DistArgs& a, cudaStream_t st) {
    const size_t sm = sizeof(DistSmem<S>);
    if (cudaFuncSetAttribute(k_dist_pair<DIST, S, STORE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) !=
        cudaSuccess)
        return -1;
    k_dist_pair<DIST, S, STORE><<<(unsigned)a.nTiles, kThreads, sm, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <int DIST, class S> int launch_pair_t(const DistArgs& a, cudaStream_t st) {
    return a.dists != nullptr ? launch_pair_s<DIST, S, true>(a, st) : launch_pair_s<DIST, S, false>(a, st);
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
    return launch_col_tiles(a.Xt, a.ld, a.dist, ListCols{a.topM, a.nproj, a.m, a.nct, a.CT},
                            (int64_t)2 * a.nproj * a.nct, a.CT, pair_tile_ctp(a.CT), a.cand, st);
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

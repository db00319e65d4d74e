// sngDbscan with independent samples (sng_findCorePoints,
// src/sDbscan.cpp:416-504, when every point's generator is seeded apart: the
// reference seeds each point from the clock when random_seed < 0, :437-440).
//
// One shared sample (the fixed-seed case, k_sng.cu) gives every sampled
// point about n reverse draws and the others none, which is not the
// reference's law when the points draw independently: then every point has S
// forward draws and about S reverse ones.  Here each block of BR = 32
// consecutive points draws its own S columns, which keeps that law (only the
// variance of the reverse count grows with the block size), and the block is
// still a dense tile: 128 draws x the block's 32 points.
//
// Draw j of block b: q = floor(hi32(splitmix64(splitmix64(seed) + b S + j)) n
// / 2^32), generated in the kernel (no draw array); a draw equal to the point
// itself is skipped.  Per pass (p, q), dist <= eps, both directions count once
// per draw (repeats counted, :459-464).  The pass bits are kept as one 32-bit
// word per (block, draw) over the block's points; the union-find and border
// passes walk the words.
//
// The distance tile is the packed FP32 tile (k_sng_pair.cu) or, for JS and
// where its column copy does not fit in memory, the scalar one here: every
// distance is the CPU path's bits, so the result equals the oracle's
// restatement of the same rule (orc_fit_sngdbscan_blocks).
#include "dist_tile.cuh"
#include "sng_draws.cuh"
#include "uf.cuh"

#include <algorithm>
#include <climits>

namespace sdb {
namespace {

using namespace dtile;

constexpr int BR = kSngBlockRows;            // points per sampled block
constexpr int BTX = 8, BCN = 4, BNT = 16 * BTX;  // 128 draws x 32 points on 128 threads

size_t tile_smem() {
    return sizeof(float) * (STAGES * (TM + BTX * BCN) * LDS) + sizeof(int) * (TM + BTX * BCN);
}

// One tile (block b, draws dt * 128 ..) per CTA.  Tiles of a block are
// consecutive: the block's 32 rows stay in L1/L2 while its draws stream past.
// EMIT (sngOptics): the pass is repeated and every passing pair goes into
// both points' tables instead of the pass words and degrees.
template <int DIST, bool EMIT>
__global__ void __launch_bounds__(BNT, 4) k_sngb_tile(SngBlockArgs a) {
    extern __shared__ __align__(16) float sm[];
    float* As = sm;                              // STAGES x TM x LDS (the draws)
    float* Bs = As + STAGES * TM * LDS;          // STAGES x 32 x LDS (the block's points)
    int* rowPoint = reinterpret_cast<int*>(Bs + STAGES * (BTX * BCN) * LDS);
    int* colPoint = rowPoint + TM;
    __shared__ uint32_t sword[TM];
    __shared__ int colCount[BR];
    __shared__ int passTotal;

    const int tid = threadIdx.x;
    const int64_t nT = (a.S + TM - 1) / TM;
    const int64_t b = (int64_t)blockIdx.x / nT;
    const int64_t j0 = ((int64_t)blockIdx.x % nT) * TM;
    for (int r = tid; r < TM; r += BNT) {
        const int64_t j = j0 + r;
        rowPoint[r] = j < a.S ? block_draw(a.key, a.S, b, j, a.n) : -1;
        sword[r] = 0;
    }
    if (tid < BR) {
        const int64_t p = b * BR + tid;
        colPoint[tid] = p < a.n ? (int)p : -1;
        colCount[tid] = 0;
    }
    if (tid == 0) passTotal = 0;
    __syncthreads();

    float acc[8][BCN];
    accumulate<DIST, BTX, BCN>(a.Xt, a.ld, a.d, rowPoint, colPoint, As, Bs, acc);
    int ty, tx;
    tile_coords<BTX>(tid, ty, tx);
    int colPass[BCN] = {0, 0, 0, 0};
    int myPass = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = ty + 16 * i;
        const int q = rowPoint[row];
        uint32_t bits = 0;
#pragma unroll
        for (int jj = 0; jj < BCN; ++jj) {
            const int col = tx + BTX * jj;
            const int p = colPoint[col];
            const float dist = finish<DIST>(acc[i][jj]);
            const bool pass = q >= 0 && p >= 0 && p != q && dist <= a.eps;
            if (pass) {
                if (EMIT) {
                    hash_insert(a, p, q, dist);
                    hash_insert(a, q, p, dist);
                }
                bits |= 1u << col;
                colPass[jj] += 1;
                ++myPass;
            }
        }
        if (!EMIT && bits) atomicOr(&sword[row], bits);
    }
    if constexpr (!EMIT) {
#pragma unroll
        for (int jj = 0; jj < BCN; ++jj)
            if (colPass[jj]) atomicAdd(&colCount[tx + BTX * jj], colPass[jj]);
        const int wp = warp_sum(myPass);
        if ((tid & 31) == 0 && wp) atomicAdd(&passTotal, wp);
        __syncthreads();
        for (int r = tid; r < TM; r += BNT) {
            const int64_t j = j0 + r;
            if (j >= a.S) continue;
            const uint32_t w = sword[r];
            a.words[b * a.S + j] = w;
            if (w) atomicAdd(a.degree + rowPoint[r], __popc(w));  // the draw's side: once per passing point
        }
        if (tid < BR && colCount[tid]) atomicAdd(a.degree + colPoint[tid], colCount[tid]);  // the points' side
        if (tid == 0 && passTotal) atomicAdd(a.pairs, (unsigned long long)passTotal);
    }
}

__global__ void k_sngb_core(SngBlockArgs a, int minPts, uint8_t* __restrict__ core) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < a.n) core[p] = a.degree[p] >= minPts - 1 ? 1 : 0;
}

// Before the union, as k_sng_hook: a warp per block of points, a point per
// lane; the point looks for three passing core draws among 64 words.
__global__ void __launch_bounds__(256) k_sngb_hook(SngBlockArgs a, const uint8_t* __restrict__ core, int32_t* parent,
                                                   int64_t j0) {
    const int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = (int)lane_id();
    const int64_t p = b * BR + lane;
    if (p >= a.n || !core[p]) return;
    RootSpan span(round_root(parent, (int)p, a.n));
    int seen = 0;
    for (int64_t j = j0; j < min(j0 + 64, a.S) && seen < 3; ++j) {
        if (!((__ldg(a.words + b * a.S + j) >> lane) & 1u)) continue;
        const int q = block_draw(a.key, a.S, b, j, a.n);
        if (!core[q]) continue;
        span.see(round_root(parent, q, a.n));
        ++seen;
    }
    span.hook(parent);
}

// The cluster passes: a warp per (block, kSpan of its words), a point of the
// block per lane with its root in a register.  32 words at a time, a lane finds
// one word's draw and that draw's root; the warp then steps through the words
// that matter.  (A thread per word with a find on both sides of every pass:
// 40 M passes at 200K x 784, p = 0.01, 3.5 ms for union and border, 0.6 here
// with the hooking rounds.)
constexpr int kSpan = 256;

struct DrawWord {
    uint32_t w;  // pass bits over the block's points
    int q;       // the draw
};
__device__ __forceinline__ DrawWord draw_word(const SngBlockArgs& a, int64_t b, int64_t j) {
    DrawWord d{0u, -1};
    if (j < a.S) {
        d.w = __ldg(a.words + b * a.S + j);
        if (d.w) d.q = block_draw(a.key, a.S, b, j, a.n);
    }
    return d;
}

// Union of every passing core-core pair.  A root in a register is an ancestor
// for good, so equality proves the same set.
__global__ void __launch_bounds__(256) k_sngb_union(SngBlockArgs a, const uint8_t* __restrict__ core,
                                                    int32_t* parent) {
    const int64_t spans = (a.S + kSpan - 1) / kSpan;
    const int64_t id = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t b = id / spans, j0 = id % spans * kSpan;
    if (b * BR >= a.n) return;
    const int lane = (int)lane_id();
    const int64_t p = b * BR + lane;
    int rp = p < a.n && core[p] ? find_root(parent, (int)p) : -1;
    for (int64_t j = j0; j < min(j0 + kSpan, a.S); j += 32) {
        const DrawWord d = draw_word(a, b, j + lane);
        const int mine = d.q >= 0 && core[d.q] ? find_root(parent, d.q) : -1;
        for (unsigned left = __ballot_sync(0xffffffffu, mine >= 0); left; left &= left - 1) {
            const int t = __ffs((int)left) - 1;
            const uint32_t w = __shfl_sync(0xffffffffu, d.w, t);
            const int rq = __shfl_sync(0xffffffffu, mine, t);
            if (rp >= 0 && rq != rp && (w >> lane) & 1u) {
                unite(parent, rp, rq);
                rp = find_root(parent, rp);
            }
        }
    }
}

// Border minima (parents of core points are roots by now): a non-core point
// takes the smallest root among its passing core neighbours, either side.
__global__ void __launch_bounds__(256) k_sngb_border(SngBlockArgs a, const uint8_t* __restrict__ core,
                                                     const int32_t* __restrict__ parent, int32_t* border) {
    const int64_t spans = (a.S + kSpan - 1) / kSpan;
    const int64_t id = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t b = id / spans, j0 = id % spans * kSpan;
    if (b * BR >= a.n) return;
    const int lane = (int)lane_id();
    const int64_t p = b * BR + lane;
    const bool pc = p < a.n && core[p];
    const int rp = pc ? __ldcg(parent + p) : INT_MAX;
    const unsigned cores = __ballot_sync(0xffffffffu, pc);  // the block's core points
    int best = INT_MAX;
    for (int64_t j = j0; j < min(j0 + kSpan, a.S); j += 32) {
        const DrawWord d = draw_word(a, b, j + lane);
        const bool qc = d.q >= 0 && core[d.q];
        const int mine = qc ? __ldcg(parent + d.q) : INT_MAX;
        // a core draw matters to non-core points, any other draw to core ones
        const bool matters = d.q >= 0 && (qc ? d.w & ~cores : d.w & cores) != 0u;
        for (unsigned left = __ballot_sync(0xffffffffu, matters); left; left &= left - 1) {
            const int t = __ffs((int)left) - 1;
            const bool pass = (__shfl_sync(0xffffffffu, d.w, t) >> lane) & 1u;
            const int rq = __shfl_sync(0xffffffffu, mine, t);
            if (rq != INT_MAX) {
                if (pass && !pc) best = min(best, rq);
            } else {
                const int r = __reduce_min_sync(0xffffffffu, pass ? rp : INT_MAX);
                const int q = __shfl_sync(0xffffffffu, d.q, t);
                if (lane == 0 && r != INT_MAX) atomicMin(border + q, r);
            }
        }
    }
    if (best != INT_MAX) atomicMin(border + p, best);
}

// Hash table sizes: a power of two >= 2 x the point's passes with repeats.
__global__ void k_sngb_caps(SngBlockArgs a, int64_t* __restrict__ cap) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > a.n) return;
    int64_t c = 0;
    if (p < a.n && a.degree[p] > 0) {
        c = 2;
        while (c < 2 * (int64_t)a.degree[p]) c <<= 1;
    }
    cap[p] = c;
}

// Distinct neighbours per point (sngOptics, src/sDbscan.cpp:1537-1541): the
// filled slots of its table; degree = their count, core >= minPts - 1.
__global__ void k_sngb_distinct(SngBlockArgs a, int minPts, int32_t* __restrict__ distinct,
                                uint8_t* __restrict__ core) {
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned l = threadIdx.x & 31u;
    if (p >= a.n) return;
    int c = 0;
    for (int64_t t = a.hashOff[p] + l; t < a.hashOff[p + 1]; t += 32) c += a.hashId[t] >= 0;
    c = warp_sum(c);
    if (l == 0) {
        distinct[p] = c;
        core[p] = c >= minPts - 1 ? 1 : 0;
    }
}

// The tables compacted into the CSR lists (nbOff from a scan of distinct).
__global__ void k_sngb_compact(SngBlockArgs a, const int64_t* __restrict__ nbOff, int32_t* __restrict__ nbIdx,
                               float* __restrict__ nbDist) {
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned l = threadIdx.x & 31u;
    if (p >= a.n) return;
    int64_t out = nbOff[p];
    for (int64_t t0 = a.hashOff[p]; t0 < a.hashOff[p + 1]; t0 += 32) {
        const int64_t t = t0 + l;
        const bool have = t < a.hashOff[p + 1] && a.hashId[t] >= 0;
        const unsigned m = __ballot_sync(0xffffffffu, have);
        if (have) {
            const int64_t o = out + __popc(m & ((1u << l) - 1u));
            nbIdx[o] = a.hashId[t];
            nbDist[o] = a.hashDist[t];
        }
        out += __popc(m);
    }
}

template <int DIST, bool EMIT> int launch_tile_t(const SngBlockArgs& a, cudaStream_t st) {
    const size_t sm = tile_smem();
    if (cudaFuncSetAttribute(k_sngb_tile<DIST, EMIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) !=
        cudaSuccess)
        return -1;
    const int64_t nb = (a.n + BR - 1) / BR, nT = (a.S + TM - 1) / TM;
    const int64_t tiles = nb * nT;
    if (tiles <= 0) return 0;
    if (tiles > (int64_t)INT_MAX) return -1;
    k_sngb_tile<DIST, EMIT><<<(unsigned)tiles, BNT, sm, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

template <bool EMIT> int launch_tiles(const SngBlockArgs& a, cudaStream_t st) {
    if (!EMIT && a.colCopy != nullptr) return launch_sngb_pair(a, st);
    if (EMIT && a.dists != nullptr) return launch_sngb_insert(a, st);
    switch (a.dist) {
        case DIST_COSINE: return launch_tile_t<DIST_COSINE, EMIT>(a, st);
        case DIST_L1: return launch_tile_t<DIST_L1, EMIT>(a, st);
        case DIST_L2: return launch_tile_t<DIST_L2, EMIT>(a, st);
        case DIST_CHI2: return launch_tile_t<DIST_CHI2, EMIT>(a, st);
        case DIST_JS: return launch_tile_t<DIST_JS, EMIT>(a, st);
    }
    return -1;
}

unsigned grid_spans(const SngBlockArgs& a) {
    const int64_t warps = (int64_t)((a.n + BR - 1) / BR) * ((a.S + kSpan - 1) / kSpan);
    return (unsigned)((warps + 7) / 8);
}

}  // namespace

int sng_block_rows() { return BR; }

int launch_sngb_pass(const SngBlockArgs& a, int minPts, uint8_t* core, cudaStream_t st) {
    const int r = launch_tiles<false>(a, st);
    if (r < 0) return -1;
    k_sngb_core<<<(a.n + 255) / 256, 256, 0, st>>>(a, minPts, core);
    return cudaPeekAtLastError() == cudaSuccess ? r + 1 : -1;
}

int launch_sngb_union(const SngBlockArgs& a, const uint8_t* core, int32_t* parent, cudaStream_t st) {
    int launches = 4;
    for (int t = 0; t < 3; ++t) {
        k_sngb_hook<<<(a.n + 255) / 256, 256, 0, st>>>(a, core, parent, 64 * t);
        const int r = launch_uf_compress_round(a.n, core, parent, st);
        if (r < 0) return -1;
        launches += r;
    }
    k_sngb_union<<<grid_spans(a), 256, 0, st>>>(a, core, parent);
    return cudaPeekAtLastError() == cudaSuccess ? launches : -1;
}

int launch_sngb_border(const SngBlockArgs& a, const uint8_t* core, const int32_t* parent, int32_t* border,
                       cudaStream_t st) {
    k_sngb_border<<<grid_spans(a), 256, 0, st>>>(a, core, parent, border);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

// sngOptics: table sizes from the pass's degrees (cap: n + 1 entries, scanned
// by the caller into hashOff), then the emitting pass into the tables.
int launch_sngb_caps(const SngBlockArgs& a, int64_t* cap, cudaStream_t st) {
    k_sngb_caps<<<(a.n + 1 + 255) / 256, 256, 0, st>>>(a, cap);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_sngb_emit(const SngBlockArgs& a, cudaStream_t st) { return launch_tiles<true>(a, st); }

int launch_sngb_distinct(const SngBlockArgs& a, int minPts, int32_t* distinct, uint8_t* core, cudaStream_t st) {
    k_sngb_distinct<<<(a.n + 7) / 8, 256, 0, st>>>(a, minPts, distinct, core);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_sngb_compact(const SngBlockArgs& a, const int64_t* nbOff, int32_t* nbIdx, float* nbDist, cudaStream_t st) {
    k_sngb_compact<<<(a.n + 7) / 8, 256, 0, st>>>(a, nbOff, nbIdx, nbDist);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace sdb

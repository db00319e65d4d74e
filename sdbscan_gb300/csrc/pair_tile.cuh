// The packed FP32 distance tile: computeDist (src/Utilities.h:212-287) for up
// to PairShape::TM gathered member rows x PairShape::CT candidate columns.
//
// Two columns share one 64-bit register pair and one packed instruction
// (fma / add / mul .rn.f32x2, each half rounded on its own): a row's value is
// broadcast to both halves, so every pair's chain is still one rounding per
// dimension in ascending order, bit-identical to the scalar tile and the CPU.
//
// Why this shape (Cosine, 784 dimensions, gathered rows, one GB300):
//  - The scalar 8 x 5 tile of dist_tile.cuh is bound by register-file
//    operands: its FMA pipe stays at 54 % and 40 TFLOP/s.  A packed FMA reads
//    the row value once for two columns: 8 x 10 and 8 x 8 tiles per thread
//    reach 52-61 TFLOP/s of the same work.
//  - Four warps per CTA, three CTAs per SM: the schedulers get the same
//    number of warps.  Five-warp CTAs (160 threads, the natural split of 50
//    columns) leave two of four schedulers with a warp less: 40-44 TFLOP/s.
//    So 50 and 40 columns use 30 of a warp's 32 lanes (6 rows x 5 column
//    groups), 192 rows per CTA; 64 and 32 columns use all of them.
//  - 32 dimensions per stage in two stages: 56 TFLOP/s against 52 for 16 in
//    three and 48 for 8 in four (a barrier per stage).
//
// The candidate tile is read from a dimension-major copy (launch_cand_tiles:
// column tile after column tile, dimension after dimension, CTP floats each),
// so a stage of it is one contiguous run and the packed column pairs need no
// shuffling; for L1 / L2 the copy is negated (a - b = a + (-b), exactly).
#pragma once

#include "dist_tile.cuh"
#include "f32x2.cuh"
#include "quotients.cuh"

namespace sdb {
namespace ptile {

constexpr int kThreads = 128;        // four warps
constexpr int KT = 32;               // dimensions per stage
constexpr int LDA = KT + 4;          // row stride of the staged rows (conflict-free 16-byte reads)
constexpr int NST = 2;               // stages

// The general Chi2 term, the form of tiles with an entry in (0, kChi2Small).
constexpr int DIST_CHI2_ANY = 5;

// One dimension of two pairs: a the row's value in both halves (negated for
// Chi2), b the two columns' values (negated but for Cosine).
template <int DIST> __device__ __forceinline__ u64 step2(u64 acc, u64 a, u64 b) {
    if (DIST == DIST_COSINE) return fma2(a, b, acc);
    if (DIST == DIST_CHI2) return add2(acc, chi2_terms(a, b));
    if (DIST == DIST_CHI2_ANY) {
        float a0, a1, b0, b1, c0, c1;
        unpack2(a, a0, a1);
        unpack2(b, b0, b1);
        unpack2(acc, c0, c1);
        return pack2(dtile::acc_step<DIST_CHI2>(c0, -a0, -b0), dtile::acc_step<DIST_CHI2>(c1, -a1, -b1));
    }
    const u64 t = add2(a, b);
    if (DIST == DIST_L2) return fma2(t, t, acc);
    float tl, th, cl, ch;  // L1
    unpack2(t, tl, th);
    unpack2(acc, cl, ch);
    return pack2(__fadd_rn(cl, fabsf(tl)), __fadd_rn(ch, fabsf(th)));
}

// TX column groups of CN columns, 32 / TX row lanes per warp, up to RMAX rows
// per thread.
template <int TX_, int CN_, int RMAX_> struct PairShape {
    static constexpr int TX = TX_, CN = CN_, RMAX = RMAX_;
    static constexpr int CT = TX * CN;                // columns
    static constexpr int CTP = (CT + 3) / 4 * 4;      // floats per dimension of the candidate copy
    static constexpr int WR = 32 / TX;                // row lanes per warp
    static constexpr int RG = 4 * WR;                 // row groups: row = group + RG i
    static constexpr int TM = RG * RMAX;              // rows
    static constexpr int NQ = CN / 4, NP = CN % 4 / 2;  // 16-byte and 8-byte fragment loads per dimension
    static constexpr size_t stage_floats = (size_t)TM * LDA + (size_t)KT * CTP;
    // the thread's row group and column group (lanes past WR * TX repeat the last one's work)
    static __device__ __forceinline__ void coords(int tid, int& rg, int& tx) {
        const int lane = min(tid & 31, WR * TX - 1);
        rg = (tid >> 5) * WR + lane / TX;
        tx = lane % TX;
    }
    static __device__ __forceinline__ bool active(int tid) { return (tid & 31) < WR * TX; }
    // first of the two columns of packed accumulator j
    static __device__ __forceinline__ int column(int tx, int j) {
        return j < 2 * NQ ? (j >> 1) * 4 * TX + 4 * tx + 2 * (j & 1) : NQ * 4 * TX + 2 * tx;
    }
};

// acc[i][j]: accumulated terms of row rg + RG i and the two columns from
// column(tx, j).  rowPoint names a point for every row below RG * RM (any
// valid point where the row is not used); cand is the tile's candidate copy;
// ld a multiple of 4.  As / Bs: NST stages of S::TM x LDA and KT x CTP floats.
// Ends with every copy landed; the caller synchronises before reusing them.
template <int DIST, class S, int RM>
__device__ __forceinline__ void pair_accumulate(const float* __restrict__ Xt, int ld, const int* rowPoint,
                                                const float* __restrict__ cand, float* As, float* Bs,
                                                u64 (&acc)[RM][S::CN / 2]) {
    const int tid = threadIdx.x;
    const int nk = (ld + KT - 1) / KT;
    auto load_stage = [&](int kc) {
        float* as = As + (kc & 1) * S::TM * LDA;
        float* bs = Bs + (kc & 1) * KT * S::CTP;
        const int k0 = kc * KT, kn = min(KT, ld - k0);
        const int c4 = (tid & 7) * 4, r0 = tid >> 3;
        if (c4 < kn) {
#pragma unroll
            for (int t = 0; t < S::RG * RM / 16; ++t) {
                const int row = r0 + 16 * t;
                dtile::cp_async16(as + row * LDA + c4, Xt + (size_t)rowPoint[row] * ld + k0 + c4, true);
            }
        }
        const float* src = cand + (size_t)k0 * S::CTP;
        for (int i = tid * 4; i < kn * S::CTP; i += kThreads * 4) dtile::cp_async16(bs + i, src + i, true);
    };
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < S::CN / 2; ++j) acc[i][j] = 0ull;
    int rg, tx;
    S::coords(tid, rg, tx);
    load_stage(0);
    dtile::cp_async_commit();
    for (int kc = 0; kc < nk; ++kc) {
        dtile::cp_async_wait<0>();
        __syncthreads();
        if (kc + 1 < nk) load_stage(kc + 1);
        dtile::cp_async_commit();
        const float* as = As + (kc & 1) * S::TM * LDA + rg * LDA;
        const float* bs = Bs + (kc & 1) * KT * S::CTP;
        const int kn = min(KT, ld - kc * KT);
        auto four_dims = [&](int kk) {
            float4 av[RM];
#pragma unroll
            for (int i = 0; i < RM; ++i) av[i] = *reinterpret_cast<const float4*>(as + i * S::RG * LDA + kk);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float* br = bs + (kk + u) * S::CTP;
                u64 b[S::CN / 2];
#pragma unroll
                for (int q = 0; q < S::NQ; ++q) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(br + q * 4 * S::TX + 4 * tx);
                    b[2 * q] = v.x;
                    b[2 * q + 1] = v.y;
                }
                if (S::NP) b[S::CN / 2 - 1] = *reinterpret_cast<const u64*>(br + S::NQ * 4 * S::TX + 2 * tx);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    const float a = u == 0 ? av[i].x : u == 1 ? av[i].y : u == 2 ? av[i].z : av[i].w;
                    const u64 a2 = pack2(a, a);
#pragma unroll
                    for (int j = 0; j < S::CN / 2; ++j) acc[i][j] = step2<DIST>(acc[i][j], a2, b[j]);
                }
            }
        };
        if (DIST == DIST_CHI2 || DIST == DIST_CHI2_ANY) {
            // a dimension at a time: four would be 30 KB of instructions
#pragma unroll 1
            for (int kk = 0; kk < kn; ++kk) {
                const float* br = bs + kk * S::CTP;
                u64 b[S::CN / 2];
#pragma unroll
                for (int q = 0; q < S::NQ; ++q) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(br + q * 4 * S::TX + 4 * tx);
                    b[2 * q] = v.x;
                    b[2 * q + 1] = v.y;
                }
                if (S::NP) b[S::CN / 2 - 1] = *reinterpret_cast<const u64*>(br + S::NQ * 4 * S::TX + 2 * tx);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    const float a = -as[i * S::RG * LDA + kk];
                    const u64 a2 = pack2(a, a);
#pragma unroll
                    for (int j = 0; j < S::CN / 2; ++j) acc[i][j] = step2<DIST>(acc[i][j], a2, b[j]);
                }
            }
            continue;
        }
        // Cosine's widest tile unrolls a whole stage (30.0 against 32.7 ms at
        // 1M x 784) where enough stages follow to pay for fetching 27 KB of
        // instructions (50K x 128: 0.25 ms unrolled, 0.23 in the loop).  L1 /
        // L2 have twice the instructions per dimension: unrolled they miss the
        // instruction cache (150K x 256, m = 100: 7.2 against 5.1 ms).
        if (DIST == DIST_COSINE && RM == S::RMAX && kn == KT && nk >= 8) {
#pragma unroll
            for (int kk = 0; kk < KT; kk += 4) four_dims(kk);
        } else {
#pragma unroll 2
            for (int kk = 0; kk < kn; kk += 4) four_dims(kk);
        }
    }
    dtile::cp_async_wait<0>();
}

}  // namespace ptile
}  // namespace sdb

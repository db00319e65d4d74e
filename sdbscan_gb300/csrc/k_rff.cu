// Random Fourier features for L1 / L2 (src/sDbscan.cpp:22-28, :59-64):
//   v = R x  (R: h x d, h = ker/2),   embed = [cos v, sin v].
// FP32 GEMM, one fmaf per dimension in ascending order per output (the
// order of the oracle's matrix-vector product), on the packed tile of
// pair_tile.cuh: a CTA takes 128 points x 64 rows of R from a dimension-major
// copy of R (launch_rff_tiles, made with the upload of R).
//
// Bound: the FP32 FMA pipe and the tile's shared-memory reads.  CTAs of one row
// tile are neighbours in the launch, so X leaves DRAM once.  The values of v go
// through shared memory before the sine and cosine: one copy of sincosf's
// instructions instead of one per accumulator, and whole 128-byte stores.
// 150K x 256, h = 512: 0.76 ms (52 TFLOP/s), against 0.96 for a scalar 8 x 4
// tile with sixteen-lane stores.
#include "pair_block.cuh"

namespace sdb {
namespace {

using namespace ptile;
using RffShape = Shape64;
constexpr int LDV = RffShape::CT + 4;  // row stride of the staged values
static_assert(RffShape::TM * LDV <= NST * RffShape::TM * LDA, "the values take the staged rows' memory");

struct RffSmem {
    float As[NST * RffShape::TM * LDA];
    float Bs[NST * KT * RffShape::CTP];
    int row[RffShape::TM];
};

// Rows of R as the tile's columns.
struct RffCols {
    int h;
    __device__ int operator()(int64_t t, int j) const {
        const int64_t r = t * RffShape::CT + j;
        return r < h ? (int)r : -1;
    }
};

__global__ void __launch_bounds__(kThreads, 3)
    k_rff(const float* __restrict__ X, int ld, int n, const float* __restrict__ Rtiles, int h, int nct,
          float* __restrict__ E, const int32_t* __restrict__ gate) {
    if (gate != nullptr && __ldg(gate) == 0) return;  // the tensor-core embedding succeeded
    extern __shared__ __align__(16) unsigned char raw[];
    RffSmem& sm = *reinterpret_cast<RffSmem*>(raw);
    const int tid = threadIdx.x;
    const int ct = blockIdx.x % nct;
    const int64_t p0 = (int64_t)(blockIdx.x / nct) * RffShape::TM;
    for (int i = tid; i < RffShape::TM; i += kThreads) sm.row[i] = (int)min(p0 + i, (int64_t)n - 1);
    __syncthreads();
    u64 acc[RffShape::RMAX][RffShape::CN / 2];
    pair_accumulate<DIST_COSINE, RffShape, RffShape::RMAX>(X, ld, sm.row, Rtiles + (size_t)ct * ld * RffShape::CTP,
                                                           sm.As, sm.Bs, acc);
    __syncthreads();
    int rg, tx;
    RffShape::coords(tid, rg, tx);
#pragma unroll
    for (int i = 0; i < RffShape::RMAX; ++i)
#pragma unroll
        for (int j = 0; j < RffShape::CN / 2; ++j)
            *reinterpret_cast<u64*>(sm.As + (rg + RffShape::RG * i) * LDV + RffShape::column(tx, j)) = acc[i][j];
    __syncthreads();
    const int c = tid & (RffShape::CT - 1), r = ct * RffShape::CT + c;
    if (r >= h) return;
    const int rows = (int)min((int64_t)RffShape::TM, n - p0);
    float* e = E + (size_t)p0 * 2 * h + r;
#pragma unroll 4
    for (int i = tid / RffShape::CT; i < rows; i += kThreads / RffShape::CT) {
        float s, co;
        sincosf(sm.As[i * LDV + c], &s, &co);
        e[(size_t)i * 2 * h] = co;
        e[(size_t)i * 2 * h + h] = s;
    }
}

int rff_col_tiles(int h) { return (h + RffShape::CT - 1) / RffShape::CT; }

}  // namespace

size_t rff_tile_floats(int h, int ld) { return (size_t)rff_col_tiles(h) * ld * RffShape::CTP; }

int launch_rff_tiles(const float* Rt, int ld, int h, float* tiles, cudaStream_t st) {
    return launch_col_tiles(Rt, ld, DIST_COSINE, RffCols{h}, rff_col_tiles(h), RffShape::CT, RffShape::CTP, tiles, st);
}

int launch_rff(const float* Xt, int ld, int n, const float* Rtiles, int h, float* E, cudaStream_t st,
               const int32_t* gate) {
    const int sm = (int)sizeof(RffSmem), nct = rff_col_tiles(h);
    if (cudaFuncSetAttribute(k_rff, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) != cudaSuccess) return -1;
    const int64_t blocks = ((int64_t)n + RffShape::TM - 1) / RffShape::TM * nct;
    k_rff<<<(unsigned)blocks, kThreads, sm, st>>>(Xt, ld, n, Rtiles, h, nct, E, gate);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace sdb

// The quotients of csrc/quotients.cuh and the terms built from them against the
// compiled division, bit for bit: counts of differences, for
// test_gpu_quotients.py.  Significands: every divisor significand (2^23 of
// them), `samples` numerators each, among them 1, the largest one and the
// divisor's own.
#include <cuda_runtime.h>

#include "dist_tile.cuh"
#include "quotients.cuh"

using namespace sdb;
typedef unsigned long long ull;

namespace {

__device__ ull hash(ull z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ float at(uint32_t significand, int exponent) {  // 2^exponent (1 + significand / 2^23)
    return ldexpf(1.0f + (float)significand * 0x1p-23f, exponent);
}
__device__ uint32_t numerator(uint32_t i, int s) {
    return s == 0 ? 0u : s == 1 ? 0x7fffffu : s == 2 ? i : (uint32_t)hash((ull)i << 8 | s) & 0x7fffffu;
}
__device__ bool differ(float a, float b) {
    return __float_as_uint(a) != __float_as_uint(b) && !(isnan(a) && isnan(b));
}

__global__ void k_row(int samples, int ec, int ex, ull* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const float c = at(i, ec);
    const RowDivisor dv = row_divisor(c);
    ull n = 0;
    for (int s = 0; s < samples; ++s) {
        const float x = at(numerator(i, s), ex) * (s & 1 ? -1.0f : 1.0f);
        n += differ(row_quotient(x, dv), __fdiv_rn(x, c));
    }
    const float special[8] = {0.0f, -0.0f, INFINITY, -INFINITY, NAN, 1e-40f, 3.4e38f, at(i, -126)};
    for (float x : special) n += differ(row_quotient(x, dv), __fdiv_rn(x, c));
    if (n) atomicAdd(bad, n);
}

// x of exponent e, s from x to 2.1 in ratio
__global__ void k_js(int samples, int e, ull* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const float x = at(i, e);
    if (x < 1e-6f || x > 1.05f) return;
    ull n = 0;
    for (int s = 0; s < samples; ++s) {
        const float u = (float)(hash((ull)i << 8 | s) >> 40) * 0x1p-24f;
        const float v = s == 0 ? x : s == 1 ? 2.1f : s == 2 ? x + x : fminf(2.1f, fmaxf(x, x * powf(2.1f / x, u)));
        n += differ(js_quotient(v, x), __fdiv_rn(v, x));
    }
    if (n) atomicAdd(bad, n);
}

// every float of [2^-23, 15], and 0
__global__ void k_log2(ull* bad, ull* tested) {
    const float l2 = 0.693147182464599609375f;
    const uint32_t first = __float_as_uint(0x1p-23f), last = __float_as_uint(15.0f);
    ull n = 0, t = 0;
    for (uint32_t b = first + blockIdx.x * blockDim.x + threadIdx.x; b <= last; b += gridDim.x * blockDim.x, ++t) {
        const float v = __uint_as_float(b);
        n += differ(js_over_l2(v), __fdiv_rn(v, l2));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) n += differ(js_over_l2(0.0f), __fdiv_rn(0.0f, l2));
    if (n) atomicAdd(bad, n);
    atomicAdd(tested, t);
}

__device__ float chi2_term(float x, float y) {
    return x > 0.0f && y > 0.0f ? __fdiv_rn(__fmul_rn(x, y), __fadd_rn(x, y)) : 0.0f;
}
__global__ void k_chi2(int samples, int ex, int ey, ull* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const float x = fminf(1.0f, at(i, ex));
    ull n = 0;
    for (int s = 0; s < samples; ++s) {
        const float y = fminf(1.0f, at(numerator(i, s), ey));
        const float x1 = s % 5 == 3 ? 0.0f : x, y1 = s % 5 >= 3 ? 0.0f : y;  // the other half: with zeros
        float q0, q1;
        unpack2(chi2_terms(pack2(-x, -x1), pack2(-y, -y1)), q0, q1);
        n += differ(q0, chi2_term(x, y)) + differ(q1, chi2_term(x1, y1));
    }
    if (n) atomicAdd(bad, n);
}

__device__ float js_step(float acc, float a, float b) {  // with the compiled division
    const float l2 = 0.693147182464599609375f;
    const float x = __fadd_rn(a, 1e-6f), y = __fadd_rn(b, 1e-6f);
    const float s = __fadd_rn(x, y);
    const float t1 = __fmul_rn(__fdiv_rn(logf(__fdiv_rn(s, x)), l2), x);
    const float t2 = __fmul_rn(__fdiv_rn(logf(__fdiv_rn(s, y)), l2), y);
    return __fadd_rn(acc, __fadd_rn(t1, t2));
}
__device__ float entry(ull z) {  // of [0, 1]: zeros, every magnitude down to subnormal ones
    const uint32_t m = (uint32_t)z & 0x7fffffu;
    const int kind = (int)(z >> 60);
    if (kind == 0) return 0.0f;
    if (kind == 1) return __uint_as_float((uint32_t)(z >> 23) % 0x3f800001u);
    return at(m, -1 - (int)((z >> 30) % 24));
}
__global__ void k_js_terms(int each, ull* bad) {
    const ull t = (ull)blockIdx.x * blockDim.x + threadIdx.x;
    ull n = 0;
    for (int s = 0; s < each; ++s) {
        const float a = entry(hash(t * each + s)), b = entry(hash(~(t * each + s)));
        n += differ(dtile::acc_step<DIST_JS>(0.0f, a, b), js_step(0.0f, a, b));
    }
    if (n) atomicAdd(bad, n);
}

__global__ void k_js_distances(const float* X, int n, int d, float* out) {
    const int p = blockIdx.y, q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    float acc = 0.0f;
    for (int j = 0; j < d; ++j) acc = js_step(acc, X[(size_t)p * d + j], X[(size_t)q * d + j]);
    out[(size_t)p * n + q] = __fsub_rn(1.0f, __fmul_rn(acc, 0.5f));
}

template <class Launch> long long count(Launch launch) {
    ull* bad = nullptr;
    if (cudaMalloc(&bad, 2 * sizeof(ull)) != cudaSuccess) return -1;
    cudaMemset(bad, 0, 2 * sizeof(ull));
    launch(bad);
    ull out[2] = {~0ull, 0};
    const bool ok = cudaMemcpy(out, bad, sizeof out, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(bad);
    return ok ? (long long)out[0] : -1;
}

constexpr unsigned kGrid = (1u << 23) / 256;

}  // namespace

extern "C" {
long long check_row(int samples, int ec, int ex) {
    return count([&](ull* b) { k_row<<<kGrid, 256>>>(samples, ec, ex, b); });
}
long long check_js(int samples, int e) {
    return count([&](ull* b) { k_js<<<kGrid, 256>>>(samples, e, b); });
}
long long check_log2() {
    return count([&](ull* b) { k_log2<<<2048, 256>>>(b, b + 1); });
}
long long check_chi2(int samples, int ex, int ey) {
    return count([&](ull* b) { k_chi2<<<kGrid, 256>>>(samples, ex, ey, b); });
}
long long check_js_terms(int each) {
    return count([&](ull* b) { k_js_terms<<<1u << 14, 256>>>(each, b); });
}
int js_distances(const float* X, int n, int d, float* out) {
    k_js_distances<<<dim3((n + 127) / 128, n), 128>>>(X, n, d, out);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
}

// The sOPTICS ordering's GPU part (formOptics_scikit, src/sDbscan.cpp:1588-1703).
//
// The outer loop takes the points in ascending order and floods from every
// core point not reached yet.  The neighbour lists are symmetric, so a flood
// reaches its start's component of the core graph -- the start being the
// component's smallest core point -- and the non-core points next to it that
// no earlier flood reached and the loop had not passed: a non-core point
// belongs to the smallest start s among its core neighbours' components if s
// is below the point itself, and stands alone otherwise.  The floods are
// therefore known beforehand and independent of one another.  Here: the
// components by union-find over the lists, every point's start, and the lists
// of the core points with renumbered neighbours and the weights
// max(core distance, distance) as order-preserving integers.
#include "uf.cuh"

#include <climits>

namespace sdb {
namespace {

// A core point hooks its root and those of four of its core neighbours
// (RootSpan; the union pass sees every edge).
__global__ void k_csr_hook(CsrArgs a, int from) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n || !a.core[p]) return;
    const int64_t e0 = a.off[p], len = a.off[p + 1] - e0;
    RootSpan span(round_root(a.parent, p, a.n));
    for (int t = from; t < from + 4 && t < len; ++t) {
        const int q = __ldg(a.idx + e0 + t);
        if (a.core[q]) span.see(round_root(a.parent, q, a.n));
    }
    span.hook(a.parent);
}

// A warp per core point over its smaller core neighbours (each edge once).  The
// paths were compressed, so two parents that agree prove the same set (a walk to
// both roots: 295 us for 5 M entries at 50K points, now 26).
__global__ void __launch_bounds__(256) k_csr_union(CsrArgs a) {
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (p >= a.n || !a.core[p]) return;
    int rp = load_parent(a.parent, p);  // compressed before: the root, or an ancestor
    for (int64_t t = a.off[p] + lane_id(); t < a.off[p + 1]; t += 32) {
        const int q = __ldg(a.idx + t);
        if (q >= p || !a.core[q]) continue;
        const int rq = load_parent(a.parent, q);  // (a common ancestor proves the same set)
        if (rq == rp) continue;
        unite(a.parent, rp, rq);
        rp = find_root(a.parent, rp);
    }
}

// The point whose turn in the outer loop emits p (p's flood's start, or p).
__global__ void k_csr_start(CsrArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    int s = p;
    if (a.core[p]) {
        s = a.parent[p];
    } else {
        for (int64_t t = a.off[p]; t < a.off[p + 1]; ++t) {
            const int q = __ldg(a.idx + t);
            if (a.core[q]) s = min(s, __ldcg(a.parent + q));
        }
    }
    a.start[p] = s;
}

__global__ void k_csr_lengths(CsrArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) a.edgeOff[a.n] = 0;
    if (p < a.n) a.edgeOff[a.newId[p]] = a.core[p] ? a.off[p + 1] - a.off[p] : 0;
}

// A warp per core point: its list at the point's new place, as far as that lies
// in [begin, end).  A neighbour of another flood becomes the point itself, which
// is done when its list is read.
__global__ void __launch_bounds__(256) k_csr_edges(CsrArgs a) {
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (p >= a.n || !a.core[p]) return;
    const int me = a.newId[p], s = a.start[p];
    const float cd = a.coreDist[p];
    const int64_t e0 = a.off[p], o = a.edgeOff[me] - e0 - a.begin;  // entry t goes to edges[o + t]
    const int64_t t0 = max(e0, -o), t1 = min(a.off[p + 1], a.end - a.begin - o);
    for (int64_t t = t0 + lane_id(); t < t1; t += 32) {
        const int q = __ldg(a.idx + t);
        const int to = __ldg(a.start + q) == s ? __ldg(a.newId + q) : me;
        a.edges[o + t] = make_uint2((uint32_t)to, key_of(fmaxf(cd, __ldg(a.dist + t))));
    }
}

}  // namespace

int launch_csr_starts(const CsrArgs& a, cudaStream_t st) {
    const int g = (a.n + 255) / 256;
    int launches = 0;
    for (int t = 0; t < 3; ++t, ++launches) {
        k_csr_hook<<<g, 256, 0, st>>>(a, 4 * t);
        const int r = launch_uf_compress_round(a.n, a.core, a.parent, st);
        if (r < 0) return -1;
        launches += r;
    }
    ClusterArgs ka{};
    ka.n = a.n;
    ka.core = a.core;
    ka.parent = a.parent;
    if (a.n < kCompressRounds && launch_uf_compress(ka, st) < 0) return -1;
    k_csr_union<<<(a.n + 7) / 8, 256, 0, st>>>(a);
    if (launch_uf_compress(ka, st) < 0) return -1;
    k_csr_start<<<g, 256, 0, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? launches + 3 : -1;
}

int launch_csr_offsets(const CsrArgs& a, int64_t* scanTmp, cudaStream_t st) {
    k_csr_lengths<<<(a.n + 255) / 256, 256, 0, st>>>(a);
    if (cudaPeekAtLastError() != cudaSuccess) return -1;
    const int r = launch_scan_i64(a.edgeOff, a.edgeOff, (size_t)a.n + 1, scanTmp, st);
    return r < 0 ? -1 : r + 1;
}

int launch_csr_edges(const CsrArgs& a, cudaStream_t st) {
    k_csr_edges<<<(a.n + 7) / 8, 256, 0, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace sdb

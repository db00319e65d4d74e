// Stage 6: cluster labels — formCluster (src/sDbscan.cpp:509-637) as a
// parallel union-find over the core graph.
//
// What the reference's BFS computes, stated without an order:
//  - cores connected through core-core edges share a cluster;
//  - clusters are numbered 0, 1, ... in increasing order of their smallest
//    core index (the outer loop visits points in ascending order, :518);
//  - a non-core point within eps of a core takes the smallest cluster id
//    among its adjacent cores (first cluster whose BFS reaches it, :603);
//  - every other point is noise (-1); n_clusters_ = clusters + 1, or 2 when
//    there is no cluster (:619, :633).
// Union-find hooks the larger root under the smaller one, so each root is
// its component's minimum index and ids follow from a prefix sum over roots.
#include "scan.cuh"
#include "uf.cuh"

#include <climits>

namespace sdb {
namespace {

__global__ void k_init(int32_t* parent, int32_t* border, int n, int keepParent) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    if (!keepParent) parent[p] = p;
    border[p] = INT_MAX;
}

// A tile of the distance stage: list l's member rows [mbeg, mend) against its
// candidate columns [CT ct, CT ct + CT) (mask word ct).
struct Tile {
    int64_t mbeg, mend;
    int ct;
    const int32_t* cand;
};

__device__ __forceinline__ bool tile_of(const ClusterArgs& a, int64_t b, Tile& tl) {
    if (b >= *a.tileTotal) return false;
    const int64_t t = tile_at(a.tilePerm, b);
    const int l = a.tileList[t];
    const int64_t ti = t - a.tileOff[l];
    const int mt = (int)(ti / a.nct);
    tl.ct = (int)(ti % a.nct);
    tl.mbeg = a.listOff[l] + (int64_t)mt * a.TM;
    tl.mend = min(tl.mbeg + a.TM, a.listOff[l + 1]);
    const int r = l % a.nproj, side = l / a.nproj;
    tl.cand = a.topM + (size_t)r * 2 * a.m + side * a.m;
    return true;
}

// Before the tile pass: rounds of hooking (RootSpan).  A core point (in an eps
// sweep one that became core this round) looks at two passing candidates of two
// of its lists and hooks the roots it sees; the tile pass sees every edge and
// restores a link that two hooks of one root lost.  With every point a set of
// its own the tile pass would send some twenty unites per point at the same few
// roots, all at once; after the rounds it finds almost nothing but equal roots
// (1M x 784: union 1827 us without, 291 + 263 for the rounds; hooking only the
// own root left 955, walking to the members' roots first 613).  In an eps sweep's
// later rounds the tile pass sees the new edges only, those hooked by among them.
__global__ void __launch_bounds__(256) k_hook(ClusterArgs a, int slot0) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n || !a.core[p] || (a.carry && a.coreEps[p] != a.round)) return;
    const bool carried = a.carry && a.round > 0;
    RootSpan span(round_root(a.parent, p, a.n, carried));
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int j = (slot0 + t) % (2 * a.k);
        const size_t at = (size_t)p * 2 * a.k + j;
        uint64_t bits = __ldg(reinterpret_cast<const unsigned long long*>(a.masks) + at * a.W);
        if (!bits) continue;
        const int32_t* cand = a.topM + (size_t)__ldg(a.topK + at) * 2 * a.m + (j >= a.k ? a.m : 0);
        for (int c = 0; c < 2 && bits; ++c, bits &= bits - 1) {
            const int q = __ldg(cand + __ffsll((long long)bits) - 1);
            if (a.core[q]) span.see(round_root(a.parent, q, a.n, carried));
        }
    }
    span.hook(a.parent);
}

// The tile's candidates of one root, as a bit set.
struct RootGroup {
    unsigned long long bits;
    int root;
};

// Union over the core-core edges of one tile.  The roots of the tile's core
// candidates are found once and the candidates grouped by root in shared
// memory; a member row then takes one step per group instead of one per
// passing candidate: it unites where the group's root differs from its own.
// A cached root is always an ancestor of its candidates (parents only move
// up), so equality proves the same set; a stale one only costs a redundant
// unite.
__global__ void __launch_bounds__(256) k_union_tiles(ClusterArgs a) {
    __shared__ RootGroup group[64];
    __shared__ int groups;
    __shared__ unsigned long long newCoreCand;  // carry: candidates that became core this round
    Tile tl;
    if (!tile_of(a, blockIdx.x, tl)) return;
    if (threadIdx.x == 0) {
        newCoreCand = 0ull;
        groups = 0;
    }
    __syncthreads();
    int q = -1;  // this thread's core candidate (threads < 64)
    if (threadIdx.x < 64) {
        const int c = tl.ct * a.CT + threadIdx.x;
        if ((int)threadIdx.x < a.CT && c < a.m) {
            q = __ldg(tl.cand + c);
            if (!a.core[q]) q = -1;
            else if (a.carry && a.coreEps[q] == a.round) atomicOr(&newCoreCand, 1ull << threadIdx.x);
        }
    }
    if (a.carry) __syncthreads();
    const int64_t row = tl.mbeg + threadIdx.x;
    int p = -1;
    uint64_t bits = 0;
    if (row < tl.mend) {
        const int2 mb = __ldg(a.members + row);
        if (a.core[mb.x]) {
            p = mb.x;
            const size_t at = ((size_t)p * 2 * a.k + mb.y) * a.W + tl.ct;
            bits = __ldg(reinterpret_cast<const unsigned long long*>(a.masks) + at);
            // carrying over a smaller eps's union-find, only edges that are new (a
            // new pair, or an endpoint that just became core) can join components
            if (a.carry && a.coreEps[p] != a.round)
                bits &= __ldg(reinterpret_cast<const unsigned long long*>(a.newMasks) + at) | newCoreCand;
        }
    }
    if (!__syncthreads_or(bits != 0)) return;  // nothing to unite in this tile
    if (threadIdx.x < 64) {
        const int root = q >= 0 ? find_root(a.parent, q) : -1;
        const unsigned same = __match_any_sync(0xffffffffu, root);
        if (root >= 0 && (int)lane_id() == __ffs((int)same) - 1) {
            RootGroup& g = group[atomicAdd(&groups, 1)];
            g.bits = (unsigned long long)same << (threadIdx.x & 32);
            g.root = root;
        }
    }
    __syncthreads();
    if (!bits) return;
    int rp = load_parent(a.parent, p);  // the root mostly; an ancestor proves the same set as well
    const int ng = groups;
    for (int g = 0; g < ng; ++g) {
        const int cr = reinterpret_cast<volatile int&>(group[g].root);
        if (cr == rp || !(bits & group[g].bits)) continue;
        unite(a.parent, rp, cr);
        rp = find_root(a.parent, rp);
        reinterpret_cast<volatile int&>(group[g].root) = rp;
    }
}

__global__ void k_compress(ClusterArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    if (a.core[p]) compress_point(a.parent, p);
}

// Border labels of one tile (parents are roots after k_compress).  A non-core
// member takes the smallest root among its passing core candidates; a non-core
// candidate takes the smallest root among the core members passing with it,
// reduced in shared memory first so each candidate sees one global atomic.  A
// core member's mask word is read only where the tile has a non-core candidate
// (1M x 784, every point core: 772 -> 181 us).
__global__ void __launch_bounds__(256) k_border_tiles(ClusterArgs a) {
    __shared__ int croot[64], cbest[64];
    __shared__ unsigned nonCore[2];  // the tile's non-core candidates
    Tile tl;
    if (!tile_of(a, blockIdx.x, tl)) return;
    int q = -1;
    if (threadIdx.x < 64) {
        const int c = tl.ct * a.CT + threadIdx.x;
        q = (int)threadIdx.x < a.CT && c < a.m ? __ldg(tl.cand + c) : -1;
        const bool core = q >= 0 && a.core[q];
        croot[threadIdx.x] = core ? __ldcg(a.parent + q) : INT_MAX;
        cbest[threadIdx.x] = INT_MAX;
        const unsigned b = __ballot_sync(0xffffffffu, q >= 0 && !core);
        if (lane_id() == 0) nonCore[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    const uint64_t nc = ((uint64_t)nonCore[1] << 32) | nonCore[0];
    const int64_t row = tl.mbeg + threadIdx.x;
    if (row < tl.mend) {
        const int2 mb = __ldg(a.members + row);
        const int p = mb.x;
        const bool core = a.core[p];
        uint64_t bits = 0;
        if (!core || nc)
            bits = __ldg(reinterpret_cast<const unsigned long long*>(a.masks) + ((size_t)p * 2 * a.k + mb.y) * a.W +
                         tl.ct);
        if (core) {
            bits &= nc;
            if (bits) {
                const int rp = __ldcg(a.parent + p);
                for (; bits; bits &= bits - 1) atomicMin(&cbest[__ffsll((long long)bits) - 1], rp);
            }
        } else {
            int best = INT_MAX;
            for (; bits; bits &= bits - 1) best = min(best, croot[__ffsll((long long)bits) - 1]);
            if (best != INT_MAX) atomicMin(a.border + p, best);
        }
    }
    if (!nc) return;
    __syncthreads();
    if (q >= 0 && cbest[threadIdx.x] != INT_MAX) atomicMin(a.border + q, cbest[threadIdx.x]);
}

// 1 for a root (a core point that is its own parent).
struct RootFlags {
    const uint8_t* core;
    const int32_t* parent;
    int n;
    __device__ int64_t operator()(size_t p) const { return p < (size_t)n && core[p] && parent[p] == (int)p ? 1 : 0; }
};

// nb > 0: rootFlag holds sums within tiles; sums the tiles' totals, which the
// block scans for itself.
__global__ void __launch_bounds__(scan::kThreads) k_labels(ClusterArgs a, const int64_t* __restrict__ sums, int nb) {
    __shared__ int64_t off[scan::kSumsInSmem];
    if (nb > 0) {
        constexpr int kPer = scan::kSumsInSmem / scan::kThreads;
        int64_t v[kPer], s = 0, total;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int t = (int)threadIdx.x * kPer + i;
            v[i] = t < nb ? __ldg(sums + t) : 0;
            s += v[i];
        }
        int64_t ex = scan::block_exclusive<scan::kThreads>(s, &total);
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            off[threadIdx.x * kPer + i] = ex;
            ex += v[i];
        }
        __syncthreads();
    }
    auto id = [&](int root) { return (int)(a.rootFlag[root] + (nb > 0 ? off[root / scan::kTile] : 0)); };
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) {
        const int c = id(a.n);
        *a.nClusters = c >= 1 ? c + 1 : 2;
    }
    if (p >= a.n) return;
    int lab = -1;
    if (a.core[p]) lab = id(a.parent[p]);
    else if (a.border[p] != INT_MAX) lab = id(a.border[p]);
    a.labels[p] = lab;
}

}  // namespace

int launch_cluster(const ClusterArgs& a, cudaStream_t st) {
    int launches = 0;
    const int g = (a.n + 255) / 256;
    k_init<<<g, 256, 0, st>>>(a.parent, a.border, a.n, a.carry && a.round > 0);
    ++launches;
    // three rounds over two lists, two candidates of each (33K x 333, 10 clusters:
    // one round over one candidate leaves the stage at 0.49 ms, three at 0.16); a
    // sweep's later rounds have few new core points
    const int rounds = !a.carry ? 3 : a.round == 0 ? 2 : 1;
    for (int t = 0; t < rounds; ++t, ++launches) {
        k_hook<<<g, 256, 0, st>>>(a, 2 * t);
        const int r = launch_uf_compress_round(a.n, a.core, a.parent, st);
        if (r < 0) return -1;
        launches += r;
    }
    k_union_tiles<<<(unsigned)a.nTiles, a.TM, 0, st>>>(a);
    ++launches;
    k_compress<<<g, 256, 0, st>>>(a);
    ++launches;
    k_border_tiles<<<(unsigned)a.nTiles, a.TM, 0, st>>>(a);
    ++launches;
    const int r = launch_cluster_labels(a, st);
    return r < 0 ? -1 : launches + r;
}

// The union-find steps for callers with their own edge kernels (sngDbscan).
int launch_uf_init(int32_t* parent, int32_t* border, int n, cudaStream_t st) {
    k_init<<<(n + 255) / 256, 256, 0, st>>>(parent, border, n, 0);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_uf_compress(const ClusterArgs& a, cudaStream_t st) {
    k_compress<<<(a.n + 255) / 256, 256, 0, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_uf_compress_round(int n, const uint8_t* core, int32_t* parent, cudaStream_t st) {
    if (n < kCompressRounds) return 0;
    ClusterArgs a{};
    a.n = n;
    a.core = core;
    a.parent = parent;
    return launch_uf_compress(a, st);
}

int launch_cluster_labels(const ClusterArgs& a, cudaStream_t st) {
    const RootFlags flags{a.core, a.parent, a.n};
    const size_t n1 = (size_t)a.n + 1, nb = scan::tiles(n1);
    // the tiles' offsets are added by the labels where a block can hold them
    const bool local = n1 > scan::kScanOne && nb <= scan::kSumsInSmem;
    const int r = local ? scan::launch_local(flags, a.rootFlag, n1, a.scanTmp, st)
                        : scan::launch(flags, a.rootFlag, n1, a.scanTmp, st);
    if (r < 0) return -1;
    k_labels<<<(a.n + scan::kThreads - 1) / scan::kThreads, scan::kThreads, 0, st>>>(a, a.scanTmp, local ? (int)nb : 0);
    return cudaPeekAtLastError() == cudaSuccess ? r + 1 : -1;
}

}  // namespace sdb

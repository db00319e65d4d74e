// sOPTICS stage: neighbour lists with distances and core distances on the
// GPU (rp_findCoreDist, src/sDbscan.cpp:1314-1474), then the ordering and
// reachability (formOptics_scikit, src/sDbscan.cpp:1588-1703).
//
// The ordering is a sequence of priority floods: each step pops the
// unprocessed point of least reachability, so a flood is inherently
// sequential, but the floods are independent of one another (k_order.cu).
// They run here in host C++, one host thread per flood at a time, over lists
// the GPU has regrouped by flood.  Ties between equal reachability values,
// which the reference's value-only heap resolves by heap order, are resolved
// by the smaller point id, so the ordering does not depend on the order of
// the neighbour lists.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <new>
#include <thread>
#include <vector>

#include "common.cuh"
#include "engine_internal.h"

namespace sdb {
int launch_core_emit(const CoreArgs& a, const void* sig, const int64_t* nbOff, int32_t* nbIdx, float* nbDist,
                     int32_t* nbFill, cudaStream_t st);
int launch_core_dist(const CoreArgs& a, const int64_t* nbOff, const float* nbDist, cudaStream_t st);
}  // namespace sdb

using namespace sdb;

namespace {

struct Edge {
    uint32_t to, key;  // neighbour's number, order-preserving key of max(core distance, distance)
};

constexpr int64_t kMinPiece = 4096;  // entries of the smallest piece that the lists come over in

constexpr uint32_t kDone = 0, kUnreached = 0xffffffffu;  // no float has these keys

// The inverse of key_of (common.cuh).
float key_value(uint32_t k) {
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    std::memcpy(&f, &u, sizeof f);
    return f;
}

struct Flood {
    int64_t entries;         // of its lists
    int first, last, start;  // its points' numbers [first, last) and the start's
};

// The floods of formOptics_scikit.  The points are numbered flood by flood
// (the outer loop's order), by point id within a flood.  best[y] is y's key:
// kUnreached, the key of its reachability while it is a seed, kDone after.
// The seed queue (Min_PQ_Pair seedSet, src/sDbscan.cpp:1609, a lazy-deletion
// heap there) is an indexed 4-ary min-heap of (key, number) words with
// decrease-key: the same pop sequence in fewer heap operations, and one
// comparison of words is the order by reachability, then id.
struct Floods {
    const int64_t* edgeOff;
    const Edge* edges;
    const int32_t* orig;  // number -> point id
    uint32_t* best;
    int32_t* pos;
    int32_t* ordering;
    float* reach;

    void run(int first, int last, int start, std::vector<uint64_t>& heap) const {
        heap.resize((size_t)(last - first));
        uint64_t* h = heap.data();
        int size = 0, out = first;
        for (int y = first; y < last; ++y) best[y] = kUnreached;
        auto relax = [&](int x) {
            const Edge* const end = edges + edgeOff[x + 1];
            for (const Edge* e = edges + edgeOff[x]; e != end; ++e) {
                const uint32_t old = best[e->to];
                if (e->key >= old) continue;  // done, or reached as near already
                best[e->to] = e->key;
                const uint64_t word = (uint64_t)e->key << 32 | e->to;
                int i = old == kUnreached ? size++ : pos[e->to];
                while (i > 0) {
                    const int par = (i - 1) >> 2;
                    if (word >= h[par]) break;
                    h[i] = h[par];
                    pos[(uint32_t)h[i]] = i;
                    i = par;
                }
                h[i] = word;
                pos[e->to] = i;
            }
        };
        best[start] = kDone;
        ordering[out++] = orig[start];
        reach[orig[start]] = kNegInfReach;
        relax(start);
        while (size > 0) {
            const uint64_t top = h[0];
            const uint64_t word = h[--size];
            if (size > 0) {
                int i = 0;
                for (int c = 1; c < size; c = 4 * i + 1) {
                    int b = c;
                    const int end = std::min(c + 4, size);
                    for (int k = c + 1; k < end; ++k)
                        if (h[k] < h[b]) b = k;
                    if (h[b] >= word) break;
                    h[i] = h[b];
                    pos[(uint32_t)h[i]] = i;
                    i = b;
                }
                h[i] = word;
                pos[(uint32_t)word] = i;
            }
            const int y = (int)(uint32_t)top;
            best[y] = kDone;
            ordering[out++] = orig[y];
            reach[orig[y]] = key_value((uint32_t)(top >> 32));
            relax(y);
        }
    }
};

}  // namespace

sdb_status sdb_engine::optics_stage(const CoreArgs& ca, int& launches) {
    cudaStream_t st = stream;
    if (!ensure(nbOff, sizeof(int64_t) * (n + 1)) || !ensure(nbFill, sizeof(int32_t) * n)) return SDB_ERR_NOMEM;
    int r = launch_scan_i32(ca.degree, n, i64(nbOff), i64(scanTmp), st);
    if (r < 0) return fail(SDB_ERR_CUDA, "scan launch failed");
    launches += r;
    int64_t total = 0;
    cudaError_t e = cudaMemcpyAsync(&total, i64(nbOff) + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "neighbour count");
    if (!ensure(nbIdx, sizeof(int32_t) * std::max<int64_t>(total, 1)) ||
        !ensure(nbDist, sizeof(float) * std::max<int64_t>(total, 1)))
        return SDB_ERR_NOMEM;
    e = cudaMemsetAsync(nbFill.ptr, 0, sizeof(int32_t) * n, st);
    if (e != cudaSuccess) return cuda_fail(e, "memset");
    r = launch_core_emit(ca, sig.ptr, i64(nbOff), i32(nbIdx), f32(nbDist), i32(nbFill), st);
    if (r < 0) return fail(SDB_ERR_CUDA, "neighbour list launch failed");
    launches += r;
    r = launch_core_dist(ca, i64(nbOff), f32(nbDist), st);
    if (r < 0) return fail(SDB_ERR_CUDA, "core distance launch failed");
    launches += r;

    return optics_order(total);
}

// The ordering and reachability from the neighbour lists of the last fit
// (nbOff / nbIdx / nbDist), core flags and core distances.  The lists' staging
// buffer is kept across fits and not zero-filled: a fresh, zeroed buffer per
// fit costs a memset and first-touch page faults over the whole list (hundreds
// of MB at 500K points) before the copy overwrites it.
// 50K x 784, 5 M list entries in ten floods: 27.9 ms for one serial flood over
// the downloaded lists, 2.8 with the floods apart (16 host cores).
sdb_status sdb_engine::optics_order(int64_t total) {
    cudaStream_t st = stream;
    cudaError_t e = cudaSuccess;
    // The lists are made: where the ordering's buffers do not fit, those that
    // only the stages before read make room (the distances are n x 2k x m
    // floats, sngOptics' tables 16 bytes an entry and more).  Where the regrouped
    // lists do not fit even then, they come over in pieces.
    auto points = [&]() {
        return ensure(parent, sizeof(int32_t) * n) && ensure(border, sizeof(int32_t) * n) &&
               ensure(floodStart, sizeof(int32_t) * n) && ensure(newId, sizeof(int32_t) * n) &&
               ensure(edgeOff, sizeof(int64_t) * (n + 1));
    };
    int64_t piece = std::max<int64_t>(total, 1);
    if (!points() || !ensure(edges, sizeof(Edge) * piece)) {
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return cuda_fail(e, "neighbour lists");
        for (DevBuf* b : {&dists, &candT, &hashIdB, &hashDistB, &sngWords}) release(*b);
        if (!points()) return SDB_ERR_NOMEM;
        while (!ensure(edges, sizeof(Edge) * piece)) {
            if (piece <= kMinPiece) return SDB_ERR_NOMEM;
            piece = std::max(kMinPiece, (piece + 1) / 2);
        }
    }
    CsrArgs a{};
    a.n = n;
    a.core = static_cast<const uint8_t*>(core.ptr);
    a.coreDist = f32(coreDist);
    a.off = i64(nbOff);
    a.idx = i32(nbIdx);
    a.dist = f32(nbDist);
    a.parent = i32(parent);
    a.start = i32(floodStart);
    a.newId = i32(newId);
    a.edgeOff = i64(edgeOff);
    a.edges = static_cast<uint2*>(edges.ptr);
    if (launch_uf_init(i32(parent), i32(border), n, st) < 0 || launch_csr_starts(a, st) < 0)
        return fail(SDB_ERR_CUDA, "flood launch failed");
    int32_t *hStart = nullptr, *hNew = nullptr, *hOrig = nullptr, *hPos = nullptr, *hFirst = nullptr;
    uint32_t* hBest = nullptr;
    int64_t* hOff = nullptr;
    Edge* hEdges = nullptr;
    try {
        int32_t* w = stageInt.get((size_t)n * 6 + 1);
        hStart = w;
        hNew = w + n;
        hOrig = w + 2 * (size_t)n;
        hPos = w + 3 * (size_t)n;
        hBest = reinterpret_cast<uint32_t*>(w + 4 * (size_t)n);
        hFirst = w + 5 * (size_t)n;
        hOff = stageOff.get((size_t)n + 1);
        hEdges = reinterpret_cast<Edge*>(stageEdge.get((size_t)std::max<int64_t>(total, 1)));
        hostOrdering.resize(n);
        hostReach.resize(n);
    } catch (const std::bad_alloc&) {
        return fail(SDB_ERR_NOMEM, "host memory for the sOPTICS neighbour lists");
    }
    e = cudaMemcpyAsync(hStart, floodStart.ptr, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "flood starts");
    // number the points by (start, id): a counting sort that keeps the ids' order
    std::fill(hFirst, hFirst + n + 1, 0);
    for (int p = 0; p < n; ++p) ++hFirst[hStart[p] + 1];
    for (int p = 0; p < n; ++p) hFirst[p + 1] += hFirst[p];
    for (int p = n - 1; p >= 0; --p) {
        const int q = --hFirst[hStart[p] + 1];
        hNew[p] = q;
        hOrig[q] = p;
    }
    e = cudaMemcpyAsync(newId.ptr, hNew, sizeof(int32_t) * n, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return cuda_fail(e, "flood numbers");
    a.end = piece;
    if (launch_csr_offsets(a, i64(scanTmp), st) < 0 || launch_csr_edges(a, st) < 0)
        return fail(SDB_ERR_CUDA, "flood list launch failed");
    e = cudaMemcpyAsync(hOff, edgeOff.ptr, sizeof(int64_t) * (n + 1), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    const int64_t kept = e == cudaSuccess ? hOff[n] : 0;
    for (int64_t at = 0; e == cudaSuccess && at < kept; at += piece) {
        if (at > 0) {
            a.begin = at;
            a.end = at + piece;
            if (launch_csr_edges(a, st) < 0) return fail(SDB_ERR_CUDA, "flood list launch failed");
        }
        e = cudaMemcpyAsync(hEdges + at, edges.ptr, sizeof(Edge) * std::min(piece, kept - at), cudaMemcpyDeviceToHost,
                            st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "neighbour list download");

    const Floods fl{hOff, hEdges, hOrig, hBest, hPos, hostOrdering.data(), hostReach.data()};
    try {
        std::vector<Flood> order;  // of more than one point
        for (int q = 0; q < n;) {
            const int s = hStart[hOrig[q]];
            int last = q + 1;
            while (last < n && hStart[hOrig[last]] == s) ++last;
            if (last == q + 1) {
                hostOrdering[q] = s;
                hostReach[s] = kNegInfReach;
            } else {
                order.push_back(Flood{hOff[last] - hOff[q], q, last, hNew[s]});
            }
            q = last;
        }
        std::sort(order.begin(), order.end(), [](const Flood& x, const Flood& y) { return x.entries > y.entries; });
        std::atomic<size_t> next{0};
        std::atomic<bool> failed{false};
        auto work = [&]() {
            try {
                std::vector<uint64_t> heap;
                for (size_t t; (t = next.fetch_add(1)) < order.size();) {
                    fl.run(order[t].first, order[t].last, order[t].start, heap);
                }
            } catch (...) {
                failed = true;
            }
        };
        // the largest floods first; a thread more for every 200K list entries
        // (starting one takes 0.06 ms), and no more than the caller's n_threads
        const unsigned most = prm.n_threads > 0 ? (unsigned)prm.n_threads
                                                : std::max(1u, std::thread::hardware_concurrency());
        const size_t threads = std::min<size_t>({(size_t)most, order.size(), (size_t)(kept / 200000) + 1, (size_t)32});
        std::vector<std::thread> helpers;
        try {
            for (size_t t = 1; t < threads; ++t) helpers.emplace_back(work);
        } catch (const std::exception&) {
            // fewer threads than wanted: the ones that started and this one do it all
        }
        work();
        for (std::thread& t : helpers) t.join();
        if (failed) return fail(SDB_ERR_NOMEM, "host memory for the sOPTICS seed queue");
    } catch (const std::bad_alloc&) {
        return fail(SDB_ERR_NOMEM, "host memory for the sOPTICS floods");
    }
    return SDB_OK;
}

// Union-find over point ids shared by the cluster stages (formCluster,
// src/sDbscan.cpp:509-637): a root is its set's smallest point id, so set
// ids follow from a prefix sum over roots.
#pragma once

#include "common.cuh"

namespace sdb {

__device__ __forceinline__ int load_parent(const int32_t* parent, int x) { return __ldcg(parent + x); }

static __device__ int find_root(int32_t* parent, int x) {
    while (true) {
        const int px = load_parent(parent, x);
        if (px == x) return x;
        const int gx = load_parent(parent, px);
        if (gx != px) parent[x] = gx;  // path halving: gx is an ancestor of x forever
        x = px;
    }
}

static __device__ void unite(int32_t* parent, int a, int b) {
    while (true) {
        a = find_root(parent, a);
        b = find_root(parent, b);
        if (a == b) return;
        if (a > b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicCAS(parent + b, b, a);
        if (old == b) return;
        b = old;
    }
}

// The root a hooking round starts from: found by walking, or, where the paths
// were compressed before the round (n >= kCompressRounds), the parent as it is
// (an ancestor if not the root).
static __device__ __forceinline__ int round_root(int32_t* parent, int x, int n) {
    return n >= kCompressRounds ? load_parent(parent, x) : find_root(parent, x);
}

// Hooking without unites: a point that saw the roots r (its own) and others of
// its component hooks the largest of them and its own under the smallest, by
// plain atomicMin.  Parents only move down, so the forest stays a forest; where
// one root is hooked twice one link is lost, so a pass over every edge has to
// follow.  (The largest as well: a root below every root it sees would
// otherwise wait for the unites.)
struct RootSpan {
    int own, lo, hi;
    __device__ explicit RootSpan(int r) : own(r), lo(r), hi(r) {}
    __device__ void see(int r) {
        lo = min(lo, r);
        hi = max(hi, r);
    }
    __device__ void hook(int32_t* parent) const {
        if (lo < own) atomicMin(parent + own, lo);
        if (lo < hi && hi != own) atomicMin(parent + hi, lo);
    }
};

}  // namespace sdb

// Union-find over point ids shared by the cluster stages (formCluster,
// src/sDbscan.cpp:509-637): a root is its set's smallest point id, so set
// ids follow from a prefix sum over roots.
#pragma once

#include "common.cuh"

namespace sdb {

__device__ __forceinline__ int load_parent(const int32_t* parent, int x) { return __ldcg(parent + x); }

// Halves the path on the way.  Where roots are linked by CAS alone (unite), a
// link once made stays and an ancestor of x is one forever.  Not so next to
// RootSpan::hook, see there.
static __device__ int find_root(int32_t* parent, int x) {
    while (true) {
        const int px = load_parent(parent, x);
        if (px == x) return x;
        const int gx = load_parent(parent, px);
        if (gx != px) parent[x] = gx;  // path halving
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

static __device__ int walk_root(const int32_t* parent, int x) {
    for (int px; (px = load_parent(parent, x)) != x;) x = px;
    return x;
}

// p's parent becomes its root.  (Each thread writes its own point only: a walk
// that halves paths would put an older ancestor over the root that another
// thread has just written, and that point would take another cluster's label.)
static __device__ void compress_point(int32_t* parent, int p) { parent[p] = walk_root(parent, p); }

// The root a hooking round starts from: found by walking, or, where the paths
// were compressed before the round (n >= kCompressRounds), the parent as it is.
// carried: links of an earlier eps hold, whose edges the union pass does not
// visit again; the walk then leaves the paths alone (below).
static __device__ __forceinline__ int round_root(int32_t* parent, int x, int n, bool carried = false) {
    return n >= kCompressRounds ? load_parent(parent, x) : carried ? walk_root(parent, x) : find_root(parent, x);
}

// Hooking without unites: a point that saw the roots r (its own) and others of
// its component hooks the largest of them and its own under the smallest, by
// plain atomicMin.  Parents only move down, so the forest stays a forest; where
// one root is hooked twice one link is lost, so a pass over every edge that the
// round hooked by has to follow.  (The largest as well: a root below every root
// it sees would otherwise wait for the unites.)
// What may be lost are links of roots only, made in this round.  But a walk
// that halves paths beside it can move a point of an older set from its root R
// to R's new parent; when R is hooked again the point and R part, and that link
// was not this round's (tests/uf_orders.cpp steps through it).  A round that
// carries older sets therefore walks without writing, and every link that is
// not a root's stays.  Dropping those rounds instead: sweeps of eight eps over
// 60K x 500 images, whose points become core late, 5.45 ms, 5.28 this way;
// 90K x 64 3.60 and 3.62.  (No halving in the other rounds either: 33K x 333
// with noise labels 1081 us, 1026 with; CAS hooks everywhere 1234.)
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

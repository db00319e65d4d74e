// The draws of sngDbscan / sngOptics with a sample per block of points
// (k_sng_blocks.cu has the rule) and the tables of distinct neighbours.
#pragma once

#include "common.cuh"

namespace sdb {

constexpr int kSngBlockRows = 32;  // points per sampled block

__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ int block_draw(uint64_t key, int64_t S, int64_t b, int64_t j, int n) {
    const uint64_t z = splitmix64(key + (uint64_t)(b * S + j));
    return (int)(((z >> 32) * (uint64_t)n) >> 32);
}

// sngOptics: q into p's open-addressing table of distinct neighbours (ids,
// -1 = empty, with the pair's distance), linear probing from a
// multiplicative hash.
__device__ __forceinline__ void hash_insert(const SngBlockArgs& a, int p, int q, float dist) {
    const int64_t o = a.hashOff[p];
    const int cap = (int)(a.hashOff[p + 1] - o);
    if (cap == 0) {
        atomicExch(a.err, 1);
        return;
    }
    uint32_t h = ((uint32_t)q * 0x9E3779B1u) & (uint32_t)(cap - 1);
    for (int probe = 0; probe < cap; ++probe, h = (h + 1) & (uint32_t)(cap - 1)) {
        const int old = atomicCAS(a.hashId + o + h, -1, q);
        if (old == -1) {  // first occurrence of q in p's list
            a.hashDist[o + h] = dist;
            return;
        }
        if (old == q) return;  // a repeat: dist(p, q) is the same value every time
    }
    atomicExch(a.err, 1);  // full table (cannot happen: cap >= 2 x the entries)
}

}  // namespace sdb

// Stage 5: neighbourhood sizes and core flags (src/sDbscan.cpp:374-400), and
// for sOPTICS the core distance (src/sDbscan.cpp:1424-1460).
//
// The reference de-duplicates each point's neighbour list, which holds both
// its own candidates within eps (A) and every point that found it within eps
// (B).  Here |A u B| = |A| + |B| - |A n B| is assembled without materialising
// the lists:
//  - |A(p)|: distinct passing candidates of p, from p's mask words; a
//    candidate met through several of p's lists is counted at its first list;
//  - |B(i)|: the distance kernel added, per tile, how many members pass
//    against candidate i (with multiplicity when a member meets i through
//    several of its lists); here each point p removes its surplus (mult - 1)
//    for every distinct candidate i;
//  - |A n B|: i in A(p) and p in A(i).  Only possible when p is itself a
//    candidate of someone ("hub"); then p in A(i) iff one of the top-m lists
//    holding p is among i's 2k lists (equal distance both ways).  Such pairs
//    are removed from B(i)'s count as well.
#include "common.cuh"

#include <algorithm>

namespace sdb {
namespace {

// true iff one of the lists point i meets through its top-k is in listMask:
// i's entries two at a time, four loads in flight (2k is even and a row starts
// on 8 bytes).
__device__ __forceinline__ bool meets_list(const CoreArgs& a, const uint32_t* listMask, int i) {
    const int2* ki = reinterpret_cast<const int2*>(a.topK + (size_t)i * 2 * a.k);
    for (int j = 0; j < a.k; j += 4) {
        int2 e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u] = __ldg(ki + min(j + u, a.k - 1));
        uint32_t hit = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j2 = 2 * min(j + u, a.k - 1);
            const int l0 = e[u].x + (j2 >= a.k ? a.nproj : 0), l1 = e[u].y + (j2 + 1 >= a.k ? a.nproj : 0);
            hit |= (listMask[l0 >> 5] >> (l0 & 31)) | (listMask[l1 >> 5] >> (l1 & 31));
        }
        if (hit & 1u) return true;
    }
    return false;
}

// true iff hub point p is in one of point i's 2k candidate lists, i.e. one
// of the top-m lists holding p is among the lists i meets through its top-k.
// Two equivalent tests; the cheaper one for p is used:
//  - p's lists (|L(p)| of them, passed in pl/np) against i's list mask
//    (kMask, one bit per list, L2-resident: only hubs have one);
//  - i's 2k top-k entries against p's list mask in shared memory.
__device__ __forceinline__ bool in_candidates_of(const CoreArgs& a, const uint32_t* listMask, const int32_t* pl,
                                                 int np, int i) {
    const int words = (2 * a.nproj + 31) / 32;
    if (np <= 2 * a.k) {
        const uint32_t* km = a.kMask + (size_t)__ldg(a.hubIdx + i) * words;
        for (int t = 0; t < np; ++t) {
            const int lst = __ldg(pl + t);
            if ((__ldg(km + (lst >> 5)) >> (lst & 31)) & 1u) return true;
        }
        return false;
    }
    return meets_list(a, listMask, i);
}

// Dense numbers (any order: they only name rows and bits) for the hubs and for
// the points that two or more lists hold.
__global__ void __launch_bounds__(256) k_hub_index(CoreArgs a, int32_t* __restrict__ hubIdx,
                                                   int32_t* __restrict__ hubPoint, int32_t* __restrict__ multiIdx,
                                                   unsigned long long* __restrict__ count) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lane = lane_id();
    const int lists = p < a.n ? (int)(a.hubOff[p + 1] - a.hubOff[p]) : 0;
    const unsigned hubs = __ballot_sync(0xffffffffu, lists > 0), multi = __ballot_sync(0xffffffffu, lists > 1);
    unsigned long long base = 0;
    if (lane < 2) {
        const int c = __popc(lane ? multi : hubs);
        if (c) base = atomicAdd(count + lane, (unsigned long long)c);
    }
    const unsigned below = (1u << lane) - 1u;
    const int h = (int)__shfl_sync(0xffffffffu, base, 0) + __popc(hubs & below);
    const int u = (int)__shfl_sync(0xffffffffu, base, 1) + __popc(multi & below);
    if (p >= a.n) return;
    hubIdx[p] = lists > 0 ? h : -1;
    multiIdx[p] = lists > 1 ? u : -1;
    if (lists > 0) hubPoint[h] = p;
}

// The hubs' list masks, a warp per hub, the mask put together in shared memory.
constexpr int kHmWarps = 8, kHmWords = 128;  // 2D <= 4096 lists
__global__ void __launch_bounds__(32 * kHmWarps) k_hub_masks(CoreArgs a, const int32_t* __restrict__ hubPoint,
                                                             const unsigned long long* __restrict__ count,
                                                             uint32_t* __restrict__ kMask) {
    __shared__ uint32_t mask[kHmWarps][kHmWords];
    const int h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (h >= (int)__ldg(count)) return;
    const int lane = (int)lane_id(), words = (2 * a.nproj + 31) / 32, slots = 2 * a.k;
    uint32_t* m = mask[threadIdx.x >> 5];
    const int32_t* tk = a.topK + (size_t)__ldg(hubPoint + h) * slots;
    for (int w = lane; w < words; w += 32) m[w] = 0u;
    __syncwarp();
    for (int j = lane; j < slots; j += 32) {
        const int l = __ldg(tk + j) + (j >= a.k ? a.nproj : 0);
        atomicOr(m + (l >> 5), 1u << (l & 31));
    }
    __syncwarp();
    for (int w = lane; w < words; w += 32) kMask[(size_t)h * words + w] = m[w];
}

// A warp per (list, word): slotMulti and slotHub = multiIdx and hubIdx of the
// slot's point, in topM's layout, and multi[l][w] bit j: the point in slot CT w + j of list l is held
// by another list too.  Most slots hold a point of one list only (about 84 % of
// the passing pairs at 1M x 784); such an occurrence is the first and only one.
__global__ void __launch_bounds__(256) k_slot_multi(const int32_t* __restrict__ topM, int D, int m, int W, int CT,
                                                    const int32_t* __restrict__ multiIdx,
                                                    const int32_t* __restrict__ hubIdx,
                                                    int32_t* __restrict__ slotMulti, int32_t* __restrict__ slotHub,
                                                    uint64_t* __restrict__ multi) {
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (q >= 2 * D * W) return;
    const int l = q / W, wd = q % W;
    const size_t row = (size_t)(l % D) * 2 * m + (l / D) * m;
    uint32_t half[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int c = h * 32 + (int)lane_id(), s = wd * CT + c;
        int u = -1;
        if (c < CT && s < m) {
            const int i = __ldg(topM + row + s);
            u = __ldg(multiIdx + i);
            slotMulti[row + s] = u;
            slotHub[row + s] = __ldg(hubIdx + i);
        }
        half[h] = __ballot_sync(0xffffffffu, u >= 0);
    }
    if (lane_id() == 0) multi[q] = ((uint64_t)half[1] << 32) | half[0];
}

// The sOPTICS emission's first occurrences.  Point p meets candidate i once per list of p
// that holds i, so with K(p) = p's 2k lists and L(i) = the top-m lists
// holding i, i's multiplicity among p's candidates is |K(p) n L(i)|, and the
// occurrence through list l is the first one iff no smaller list of
// K(p) n L(i) exists.  sig[l][s] lists, for the point in slot s of list l, the
// other lists holding it (up to three; cnt > 3 sends the test to the hub-list
// CSR), and K(p) sits as a bit mask in shared memory while p is processed.

__global__ void k_slot_sigs(const int32_t* __restrict__ topM, int D, int m, const int64_t* __restrict__ hubOff,
                            const int32_t* __restrict__ hubLists, int4* __restrict__ sig) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 2 * D * m) return;
    const int l = q / m, s = q % m, r = l % D, side = l / D;
    const int i = topM[(size_t)r * 2 * m + side * m + s];
    int o[3] = {-1, -1, -1}, c = 0;
    for (int64_t h = hubOff[i]; h < hubOff[i + 1]; ++h) {
        const int lst = hubLists[h];
        if (lst == l) continue;
        if (c < 3) o[c] = lst;
        ++c;
    }
    sig[q] = make_int4(o[0], o[1], o[2], c);
}

__device__ __forceinline__ bool has_list(const uint32_t* km, int lst) { return (km[lst >> 5] >> (lst & 31)) & 1u; }

// Multiplicity and first-occurrence test of candidate i, met through list l.
__device__ __forceinline__ void occurrence(const CoreArgs& a, const uint32_t* km, const int4* sig, int l, int s, int i,
                                          int& mult, bool& first) {
    const int4 g = __ldg(sig + (size_t)l * a.m + s);
    mult = 1;
    first = true;
    if (g.w <= 3) {
        if (g.w > 0 && has_list(km, g.x)) { ++mult; first &= g.x > l; }
        if (g.w > 1 && has_list(km, g.y)) { ++mult; first &= g.y > l; }
        if (g.w > 2 && has_list(km, g.z)) { ++mult; first &= g.z > l; }
    } else {
        for (int64_t h = a.hubOff[i]; h < a.hubOff[i + 1]; ++h) {
            const int o = a.hubLists[h];
            if (o != l && has_list(km, o)) {
                ++mult;
                first &= o > l;
            }
        }
    }
}

// Per-warp shared memory: K(p) mask and p's hub-list mask (2D bits each).
__device__ __forceinline__ void set_k_mask(uint32_t* km, int l, bool on) {
    if (on) atomicOr(km + (l >> 5), 1u << (l & 31));
}

// Visits the passing slots of point p, slot by slot; f(jj, l, s, i, first,
// mult) on lanes (the sOPTICS list emission).
template <typename F>
__device__ __forceinline__ void visit_point(const CoreArgs& a, uint32_t* km, const int4* sig, int p, F&& f) {
    const unsigned lane = lane_id();
    const int slots = 2 * a.k;
    const unsigned long long* mk64 = reinterpret_cast<const unsigned long long*>(a.masks);
    int rA = 0, rB = 0;
    uint64_t mA0 = 0, mB0 = 0;
    if ((int)lane < slots) {
        rA = __ldg(a.topK + (size_t)p * slots + lane);
        mA0 = __ldg(mk64 + ((size_t)p * slots + lane) * a.W);
    }
    if ((int)lane + 32 < slots) {
        rB = __ldg(a.topK + (size_t)p * slots + lane + 32);
        mB0 = __ldg(mk64 + ((size_t)p * slots + lane + 32) * a.W);
    }
    const int lA = rA + ((int)lane >= a.k ? a.nproj : 0), lB = rB + ((int)lane + 32 >= a.k ? a.nproj : 0);
    set_k_mask(km, lA, (int)lane < slots);
    set_k_mask(km, lB, (int)lane + 32 < slots);
    __syncwarp();
    for (int jj = 0; jj < slots; ++jj) {
        const int src = jj & 31;
        const int l = __shfl_sync(0xffffffffu, jj < 32 ? lA : lB, src);
        const int r = l % a.nproj, side = l / a.nproj;
        const int32_t* lst = a.topM + (size_t)r * 2 * a.m + side * a.m;
        for (int wd = 0; wd < a.W; ++wd) {
            uint64_t mk;
            if (wd == 0) {
                const uint64_t mine = jj < 32 ? mA0 : mB0;
                const uint32_t lo = __shfl_sync(0xffffffffu, (uint32_t)mine, src);
                const uint32_t hi = __shfl_sync(0xffffffffu, (uint32_t)(mine >> 32), src);
                mk = ((uint64_t)hi << 32) | lo;
            } else {
                mk = __ldg(mk64 + ((size_t)p * slots + jj) * a.W + wd);
            }
            if (mk) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int bit = half * 32 + (int)lane;
                    if ((mk >> bit) & 1ull) {
                        const int s = wd * a.CT + bit;
                        const int i = __ldg(lst + s);
                        int mult;
                        bool isFirst;
                        occurrence(a, km, sig, l, s, i, mult, isFirst);
                        f(jj, l, s, i, isFirst, mult);
                    }
                }
            }
        }
    }
    __syncwarp();
    if ((int)lane < slots) km[lA >> 5] = 0u;
    if ((int)lane + 32 < slots) km[lB >> 5] = 0u;
    __syncwarp();
}

__device__ __forceinline__ void mark_lists(const CoreArgs& a, uint32_t* listMask, int64_t h0, int64_t h1,
                                           int maskWords) {
    const unsigned l = lane_id();
    for (int t = (int)l; t < maskWords; t += 32) listMask[t] = 0u;
    __syncwarp();
    for (int64_t h = h0 + l; h < h1; h += 32) {
        const int lst = a.hubLists[h];
        atomicOr(&listMask[lst >> 5], 1u << (lst & 31));
    }
    __syncwarp();
}

// Per-warp shared memory of k_core_dedupe, between the seen bits and p's list mask.
constexpr int kDdHalves = 32;      // mask half-words (32 bits) per round, one per lane
constexpr int kDdLists = 8;        // lists of a hub tested against the candidates' list masks
constexpr int kDdSeenWords = 1024; // seen bits held at once: 32768 points (more are taken in passes)
struct alignas(16) DedupeWarp {
    uint32_t drop[kDdHalves];      // gathered pairs that are no first occurrence
    int32_t off[kDdHalves];        // the half-word's first slot in topM
    uint16_t item[kDdHalves * 32]; // the round's pairs that need the per-pair test: (half-word, bit)
    int32_t lists[kDdLists];       // a hub's lists, when it has at most that many
};
__host__ __device__ constexpr size_t dedupe_warp_bytes(int seenWords, int maskWords) {
    return (sizeof(uint32_t) * ((size_t)seenWords + maskWords) + sizeof(DedupeWarp) + 15) / 16 * 16;
}

// A point of at most 32 passing pairs, a pair per lane: repeats are lanes of
// the same candidate (no seen bits to clear: 150K x 256 L2, m = 100, core stage
// 266 -> 145 us).  Returns the number of distinct candidates; the point's
// output words are cleared already.  pairs: of this lane's 16-byte pieces.  (Not
// inlined: it costs the dense path registers.)
__device__ __noinline__ int dedupe_sparse(const CoreArgs& a, DedupeWarp& sw, const uint32_t* listMask, int p, int np,
                                          int pairs, int allPairs) {
    const int lane = (int)lane_id(), slots = 2 * a.k, maskWords = (2 * a.nproj + 31) / 32;
    const size_t row = (size_t)p * 2 * slots * a.W;
    const uint4* row4 = reinterpret_cast<const uint4*>(reinterpret_cast<const uint32_t*>(a.masks) + row);
    uint32_t* item = reinterpret_cast<uint32_t*>(sw.item);
    int at = pairs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
    }
    at -= pairs;
    for (int t = lane; pairs > 0; t += 32) {
        const uint4 v = __ldg(row4 + t);
        const uint32_t halves[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
            for (uint32_t b = halves[q]; b; b &= b - 1, --pairs)
                item[at++] = (uint32_t)(4 * t + q) << 5 | (uint32_t)(__ffs((int)b) - 1);
    }
    __syncwarp();
    const bool have = lane < allPairs;
    const uint32_t it = have ? item[lane] : 0u;
    const int half = (int)(it >> 5), word = half >> 1, bit = (int)(it & 31u);
    const int jj = a.W == 1 ? word : word / a.W, wd = word - jj * a.W;
    int u = -1, i = 0, h = 0;
    if (have) {
        const int off = __ldg(a.topK + (size_t)p * slots + jj) * 2 * a.m + (jj >= a.k ? a.m : 0) + wd * a.CT +
                        (half & 1) * 32 + bit;
        u = __ldg(a.slotMulti + off);
        i = __ldg(a.topM + off);
        h = np ? __ldg(a.slotHub + off) : 0;
    }
    const unsigned same = __match_any_sync(0xffffffffu, u >= 0 ? u : -2 - lane);
    const bool first = have && lane == __ffs((int)same) - 1;
    bool out1 = have && !first;
    if (first) {
        if (np <= kDdLists) {
            for (int q = 0; q < np; ++q) {
                const int l = sw.lists[q];
                out1 |= (__ldg(a.kMask + (size_t)h * maskWords + (l >> 5)) >> (l & 31)) & 1u;
            }
        } else {
            out1 = meets_list(a, listMask, i);
        }
        uint32_t* out = reinterpret_cast<uint32_t*>(a.accumulate ? a.newMasks : a.firstMasks);
        atomicOr(out + row + half, 1u << bit);
        if (a.accumulate) atomicOr(reinterpret_cast<uint32_t*>(a.firstMasks) + row + half, 1u << bit);
    }
    if (out1) atomicSub(a.inRaw + i, 1);
    const int distinct = __popc(__ballot_sync(0xffffffffu, first));
    __syncwarp();
    return distinct;
}

// Persistent warps, each over points p = warp, warp + total, ...  A candidate
// that no other list holds is a first occurrence as it stands.  The others are
// gathered into a dense per-warp list (so the warp's instructions follow those
// pairs, not every slot and lane) and set one bit each in a shared-memory bit
// row indexed by multiIdx: the occurrence that finds the bit clear is the
// first (which one it is does not matter to any later stage), every other one
// takes itself out of the candidate's count.  A hub's first occurrences need
// the in-candidates test, so all its pairs are gathered.
// (Signatures per slot tested against the point's lists, the form before, walk
// a candidate's lists where more than four hold it.  Core stage then and now:
// 2K x 64, 51 lists a point, 317 -> 62 us; 50K x 128 328 -> 211; 1M x 784
// 2147 -> 1744.)  Bound: latency, of the slot and list-mask loads in L2 and of
// the shared-memory accesses in equal parts (5.5 stalled warps per issue each at
// 200K x 784, issue slots 44 % and the shared-memory pipe 62 % used).
__global__ void __launch_bounds__(128, 8) k_core_dedupe(CoreArgs a, int seenWords) {
    extern __shared__ __align__(16) unsigned char ddShm[];
    const int w = threadIdx.x >> 5;
    const int lane = (int)lane_id();
    const int maskWords = (2 * a.nproj + 31) / 32;
    uint32_t* seen = reinterpret_cast<uint32_t*>(ddShm + (size_t)w * dedupe_warp_bytes(seenWords, maskWords));
    DedupeWarp& sw = *reinterpret_cast<DedupeWarp*>(seen + seenWords);
    uint32_t* listMask = reinterpret_cast<uint32_t*>(&sw + 1);
    const int gw = blockIdx.x * (blockDim.x >> 5) + w;
    const int nw = gridDim.x * (blockDim.x >> 5);
    const int slots = 2 * a.k;
    const int nHalves = 2 * slots * a.W;
    const uint32_t* mk32 = reinterpret_cast<const uint32_t*>(a.masks);
    const uint32_t* mu32 = reinterpret_cast<const uint32_t*>(a.multi);
    uint32_t* out = reinterpret_cast<uint32_t*>(a.accumulate ? a.newMasks : a.firstMasks);
    uint32_t* all = reinterpret_cast<uint32_t*>(a.firstMasks);
    const int multi = (int)__ldg(a.multiCount), span = seenWords * 32;
    for (int p = gw; p < a.n; p += nw) {
        const size_t row = (size_t)p * nHalves;
        // a point without a passing pair (common in a sweep round) only clears
        // its first-occurrence words (this round's words when accumulating);
        // a row is an even number of words, 16 bytes at a time
        int pairs = 0;  // this lane's passing pairs
        const uint4* row4 = reinterpret_cast<const uint4*>(mk32 + row);
        for (int t = lane; t < nHalves / 4; t += 32) {
            const uint4 v = __ldg(row4 + t);
            pairs += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
        }
        const int allPairs = warp_sum(pairs);
        if (allPairs <= 32) {
            for (int t = lane; t < nHalves / 4; t += 32)
                reinterpret_cast<uint4*>(out + row)[t] = make_uint4(0u, 0u, 0u, 0u);
        }
        if (allPairs == 0) {
            if (lane == 0) a.aCount[p] = 0;
            continue;
        }
        const int64_t h0 = a.hubOff[p];
        const int np = (int)(a.hubOff[p + 1] - h0);
        const bool hub = np > 0;
        const bool few = np <= kDdLists;
        if (few) {
            if (lane < np) sw.lists[lane] = a.hubLists[h0 + lane];
        } else {
            mark_lists(a, listMask, h0, h0 + np, maskWords);
        }
        int distinct = 0;
        if (allPairs <= 32) {
            distinct = dedupe_sparse(a, sw, listMask, p, hub ? np : 0, pairs, allPairs);
            if (lane == 0) a.aCount[p] = distinct;
            continue;
        }
        // pass s0 takes the candidates numbered [s0, s0 + span); the first one
        // takes those of a single list too
        for (int s0 = 0; s0 == 0 || s0 < multi; s0 += span) {
            for (int t = lane; 128 * t < min(span, multi - s0); t += 32)
                reinterpret_cast<uint4*>(seen)[t] = make_uint4(0u, 0u, 0u, 0u);
            for (int hb = 0; hb < nHalves; hb += kDdHalves) {
                const int g = hb + lane;  // this lane's half-word: word g / 2 of slot g / 2W
                uint32_t mk = 0, mu = 0;
                if (g < nHalves) {
                    mk = __ldg(mk32 + row + g);
                    const int word = g >> 1;
                    const int jj = a.W == 1 ? word : word / a.W, wd = word - jj * a.W;
                    const int r = __ldg(a.topK + (size_t)p * slots + jj), side = jj >= a.k;
                    sw.off[lane] = r * 2 * a.m + side * a.m + wd * a.CT + (g & 1) * 32;
                    mu = hub && s0 == 0
                             ? ~0u
                             : __ldg(mu32 + 2 * ((size_t)(r + (side ? a.nproj : 0)) * a.W + wd) + (g & 1));
                }
                const uint32_t sole = s0 == 0 ? mk & ~mu : 0u, todo = mk & mu;
                distinct += __popc(sole);
                sw.drop[lane] = 0u;
                // gather the pairs that need the test: lane-serial over its half-word's bits
                const int cnt = __popc(todo);
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                uint16_t* at = sw.item + (incl - cnt);
                for (uint32_t t = todo; t; t &= t - 1) *at++ = (uint16_t)((lane << 5) | (__ffs((int)t) - 1));
                __syncwarp();
                // two pairs per lane and step, their loads together: the loop
                // waits for L2, not for instructions
                for (int t = lane; t < total; t += 64) {
                    int it[2], u[2], i[2], h[2];
                    bool have[2], first[2], out1[2];  // out1: one to take out of the candidate's count
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        have[e] = first[e] = t + 32 * e < total;
                        it[e] = sw.item[have[e] ? t + 32 * e : t];
                        const int off = sw.off[it[e] >> 5] + (it[e] & 31);
                        u[e] = __ldg(a.slotMulti + off);
                        i[e] = __ldg(a.topM + off);
                        h[e] = hub ? __ldg(a.slotHub + off) : 0;
                        out1[e] = false;
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int b = u[e] - s0;
                        if (first[e] && u[e] >= 0) {
                            if ((unsigned)b >= (unsigned)span) {
                                first[e] = false;  // another pass's
                            } else if ((atomicOr(seen + (b >> 5), 1u << (b & 31)) >> (b & 31)) & 1u) {
                                first[e] = false;  // a repeat of a candidate already counted
                                out1[e] = true;
                            }
                        }
                        // (marking the others: neighbouring lanes' pairs share a
                        // half-word, and most are first occurrences)
                        if (first[e]) ++distinct;
                        else if (have[e]) atomicOr(&sw.drop[it[e] >> 5], 1u << (it[e] & 31));
                    }
                    if (few) {  // p in A(i): one of p's lists is among those i meets
                        const uint32_t* km0 = a.kMask + (size_t)h[0] * maskWords;
                        const uint32_t* km1 = a.kMask + (size_t)h[1] * maskWords;
                        for (int q = 0; q < np; ++q) {
                            const int l = sw.lists[q];
                            const uint32_t w0 = first[0] ? __ldg(km0 + (l >> 5)) : 0u;
                            const uint32_t w1 = first[1] ? __ldg(km1 + (l >> 5)) : 0u;
                            out1[0] |= (w0 >> (l & 31)) & 1u;
                            out1[1] |= (w1 >> (l & 31)) & 1u;
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (first[e]) out1[e] = meets_list(a, listMask, i[e]);
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (out1[e]) atomicSub(a.inRaw + i[e], 1);
                }
                __syncwarp();
                if (g < nHalves) {
                    uint32_t f = sole | (todo & ~sw.drop[lane]);
                    if (a.accumulate && f) all[row + g] |= f;
                    if (s0) f |= out[row + g];
                    out[row + g] = f;
                }
                __syncwarp();
            }
        }
        distinct = warp_sum(distinct);
        if (lane == 0) a.aCount[p] = distinct;
    }
}

// sOPTICS neighbour lists (src/sDbscan.cpp:1371-1372, :1404-1405, de-duplicated
// at :1428-1431): for every point p, its distinct candidates within eps (own
// entries, first |A(p)| slots of its row) and every point that found p within
// eps without p finding it back (in entries, after them).  Row p starts at
// nbOff[p] and holds degree[p] = |A(p)| + |B(p) \ A(p)| entries.
__global__ void k_core_emit(CoreArgs a, const int4* __restrict__ sig, const int64_t* __restrict__ nbOff,
                            int32_t* __restrict__ nbIdx, float* __restrict__ nbDist, int32_t* __restrict__ nbFill) {
    extern __shared__ uint32_t shm[];
    const int w = threadIdx.x >> 5;
    const unsigned lane = lane_id();
    const int maskWords = (2 * a.nproj + 31) / 32;
    uint32_t* km = shm + (size_t)w * (2 * maskWords + 1);
    uint32_t* listMask = km + maskWords;
    int* cursor = reinterpret_cast<int*>(listMask + maskWords);  // next own-entry slot of the row
    for (int t = (int)lane; t < maskWords; t += 32) km[t] = 0u;
    __syncwarp();
    const int gw = blockIdx.x * (blockDim.x >> 5) + w;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int p = gw; p < a.n; p += nw) {
        const int64_t h0 = a.hubOff[p], h1 = a.hubOff[p + 1];
        const bool hub = h1 > h0;
        if (hub) mark_lists(a, listMask, h0, h1, maskWords);
        if (lane == 0) *cursor = 0;
        __syncwarp();
        const int64_t row = nbOff[p];
        visit_point(a, km, sig, p, [&](int jj, int, int s, int i, bool first, int) {
            if (!first) return;
            const float dd = a.dists[((size_t)p * 2 * a.k + jj) * a.m + s];
            const int pos = atomicAdd(cursor, 1);
            nbIdx[row + pos] = i;
            nbDist[row + pos] = dd;
            if (!(hub && in_candidates_of(a, listMask, a.hubLists + h0, (int)(h1 - h0), i))) {
                const int q = atomicAdd(nbFill + i, 1);
                const int64_t at = nbOff[i] + a.aCount[i] + q;
                nbIdx[at] = p;
                nbDist[at] = dd;
            }
        });
    }
}

__global__ void k_core_finish(CoreArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    if (a.accumulate) {  // this round's pairs are new neighbours: the degree grows
        const int deg = a.degree[p] + a.aCount[p] + a.inRaw[p];
        a.degree[p] = deg;
        if (!a.core[p] && deg >= a.minPts - 1) {
            a.core[p] = 1;
            a.coreEps[p] = a.round;
        }
        return;
    }
    const int deg = a.aCount[p] + a.inRaw[p];
    a.degree[p] = deg;
    a.core[p] = deg >= a.minPts - 1 ? 1 : 0;
}

// Core distance: the (minPts-1)-th smallest distance of a core point's row
// (nth_element at minPts-2, src/sDbscan.cpp:1443-1446); 0 for other points
// (src/sDbscan.cpp:1420).  One warp per point, 4-pass radix select over the
// order-preserving keys of the distances.
__global__ void k_core_dist(CoreArgs a, const int64_t* __restrict__ nbOff, const float* __restrict__ nbDist) {
    __shared__ unsigned hist[8][256];
    const int w = threadIdx.x >> 5;
    const unsigned l = lane_id();
    const int p = blockIdx.x * (blockDim.x >> 5) + w;
    if (p >= a.n) return;
    if (!a.core[p]) {
        if (l == 0) a.coreDist[p] = 0.0f;
        return;
    }
    const int64_t r0 = nbOff[p], r1 = nbOff[p + 1];
    int need = a.minPts - 1;  // 1-based rank of the wanted value
    uint32_t prefix = 0, pmask = 0;
    unsigned* hs = hist[w];
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int b = (int)l; b < 256; b += 32) hs[b] = 0;
        __syncwarp();
        for (int64_t t = r0 + l; t < r1; t += 32) {
            const uint32_t k = key_of(nbDist[t]);
            if ((k & pmask) == prefix) atomicAdd(&hs[(k >> shift) & 255u], 1u);
        }
        __syncwarp();
        // the bucket holding the need-th smallest: eight bins a lane (one lane
        // after the other through 256: 167 us at 50K points of 99 neighbours, now
        // 71)
        int c[8], sum = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) sum += c[b] = (int)hs[8 * l + b];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)l >= o) incl += v;
        }
        const unsigned at = __ballot_sync(0xffffffffu, incl >= need);
        const int owner = at ? __ffs((int)at) - 1 : 31;
        int acc = incl - sum, pick = 8 * (int)l + 7;
#pragma unroll
        for (int b = 7; b >= 0; --b) {  // the first bin that reaches need, from behind
            int before = acc;
#pragma unroll
            for (int q = 0; q < b; ++q) before += c[q];
            if (before + c[b] >= need) pick = 8 * (int)l + b;
        }
#pragma unroll
        for (int b = 0; b < 8; ++b)
            if (8 * (int)l + b < pick) acc += c[b];
        pick = __shfl_sync(0xffffffffu, pick, owner);
        need -= __shfl_sync(0xffffffffu, acc, owner);
        prefix |= (uint32_t)pick << shift;
        pmask |= 255u << shift;
        __syncwarp();
    }
    if (l == 0) a.coreDist[p] = float_of_key(prefix);
}

}  // namespace

static int core_grid(int n, int warps) {
    const int blocks = (n + warps - 1) / warps;
    return std::min(blocks, sm_count() * 8);
}

int launch_slot_sigs(const int32_t* topM, int D, int m, const int64_t* hubOff, const int32_t* hubLists, void* sig,
                     cudaStream_t st) {
    const int total = 2 * D * m;
    k_slot_sigs<<<(total + 255) / 256, 256, 0, st>>>(topM, D, m, hubOff, hubLists, static_cast<int4*>(sig));
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_core_dedupe(const CoreArgs& a, cudaStream_t st) {
    const int warps = 4;
    // seen bits for every point that two lists can hold, whole 16 bytes
    const int64_t most = std::min<int64_t>(a.n, (int64_t)a.nproj * a.m);
    const int seenWords = (int)std::min<int64_t>(kDdSeenWords, (most + 127) / 128 * 4);
    const size_t sm = dedupe_warp_bytes(seenWords, (2 * a.nproj + 31) / 32) * warps;
    if (sm > 48 * 1024 &&
        cudaFuncSetAttribute(k_core_dedupe, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
        return -1;
    const int perSm = (int)std::max<size_t>(1, std::min<size_t>(12, 224 * 1024 / (sm + 1024)));
    const int blocks = std::min((a.n + warps - 1) / warps, sm_count() * perSm);
    k_core_dedupe<<<blocks, warps * 32, sm, st>>>(a, seenWords);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_hub_index(const CoreArgs& a, int32_t* hubIdx, int32_t* hubPoint, int32_t* multiIdx, uint32_t* kMask,
                     int32_t* slotMulti, int32_t* slotHub, uint64_t* multi, unsigned long long* count,
                     cudaStream_t st) {
    k_hub_index<<<(a.n + 255) / 256, 256, 0, st>>>(a, hubIdx, hubPoint, multiIdx, count);
    if (cudaPeekAtLastError() != cudaSuccess) return -1;
    const int64_t hubs = std::min<int64_t>(a.n, (int64_t)2 * a.nproj * a.m);
    k_hub_masks<<<(unsigned)((hubs + 7) / 8), 256, 0, st>>>(a, hubPoint, count, kMask);
    if (cudaPeekAtLastError() != cudaSuccess) return -1;
    k_slot_multi<<<(2 * a.nproj * a.W + 7) / 8, 256, 0, st>>>(a.topM, a.nproj, a.m, a.W, a.CT, multiIdx, hubIdx,
                                                              slotMulti, slotHub, multi);
    return cudaPeekAtLastError() == cudaSuccess ? 3 : -1;
}

int launch_core_finish(const CoreArgs& a, cudaStream_t st) {
    k_core_finish<<<(a.n + 255) / 256, 256, 0, st>>>(a);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_core_emit(const CoreArgs& a, const void* sig, const int64_t* nbOff, int32_t* nbIdx, float* nbDist,
                     int32_t* nbFill, cudaStream_t st) {
    const int warps = 8;
    const size_t sm = sizeof(uint32_t) * (2 * ((2 * a.nproj + 31) / 32) + 1) * warps;
    k_core_emit<<<core_grid(a.n, warps), warps * 32, sm, st>>>(a, static_cast<const int4*>(sig), nbOff, nbIdx,
                                                               nbDist, nbFill);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_core_dist(const CoreArgs& a, const int64_t* nbOff, const float* nbDist, cudaStream_t st) {
    k_core_dist<<<(a.n + 7) / 8, 256, 0, st>>>(a, nbOff, nbDist);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace sdb

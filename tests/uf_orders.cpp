// Every order of the union-find operations of csrc/uf.cuh on a few points.
//
// uf_host.h is uf.cuh with its includes taken out: int32_t cells, the cached
// load and the two atomics below stand in for device memory, each one step of
// its thread.  A state is the memory and what every thread has read so far (a
// thread is deterministic), so each is followed once; a prefix of steps is
// replayed to reach it.
//
// The case: an eps sweep's round above the first.  An old set holds the links
// of an earlier eps, three points became core, each with an edge to an old
// member.  They hook (as k_hook does), in every order; then the new edges are
// united and no others (as k_union_tiles does in a carried round).  One set has
// to be left.  Arguments: the point count that the hooking rule goes by, and 1
// for a carried round's walk, 0 for the other rounds', which halves paths.
// With one argument, compress_point instead (compress below).
#include <setjmp.h>
#include <ucontext.h>

#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <set>
#include <vector>

static void step();                 // the calling thread's turn ends
static void note(int value);        // the calling thread has read value

struct Cell {
    int v;
    Cell& operator=(int x) {
        step();
        v = x;
        return *this;
    }
};
static int __ldcg(const Cell* c) {
    step();
    note(c->v);
    return c->v;
}
static int atomicMin(Cell* c, int x) {
    step();
    const int old = c->v;
    if (x < old) c->v = x;
    note(old);
    return old;
}
static int atomicCAS(Cell* c, int expect, int x) {
    step();
    const int old = c->v;
    if (old == expect) c->v = x;
    note(old);
    return old;
}
template <class T> static T min(T a, T b) { return a < b ? a : b; }
template <class T> static T max(T a, T b) { return a < b ? b : a; }
static constexpr int kCompressRounds = KCOMPRESS;

#define __device__
#define __forceinline__ inline
#define int32_t Cell
#include "uf_host.h"
#undef int32_t

using namespace sdb;

constexpr int N = 6, kThreads = 3;
static Cell mem[N];

// ---- threads as contexts that swap back at each step -----------------------
struct Fiber {
    ucontext_t ctx;  // its start
    jmp_buf at;      // where it left off
    std::vector<char> stack = std::vector<char>(64 << 10);
    std::vector<int> reads;
    bool done = false;
};
static Fiber fibers[kThreads];
static jmp_buf home;
static int current = -1;
static std::function<void(int)> body;

static void step() {
    if (current >= 0 && !_setjmp(fibers[current].at)) _longjmp(home, 1);
}
static void note(int value) {
    if (current >= 0) fibers[current].reads.push_back(value);
}
static void entry() {
    body(current);
    fibers[current].done = true;
    _longjmp(home, 1);
}
static void turn(int t, bool first = false) {
    current = t;
    if (!_setjmp(home)) {
        if (first) setcontext(&fibers[t].ctx);
        else _longjmp(fibers[t].at, 1);
    }
    current = -1;  // outside the threads a step is just a step
}

typedef std::vector<int> Mem;

// Runs the threads in every order from start; the memories they can leave.
static std::set<Mem> outcomes(const Mem& start) {
    std::set<Mem> out;
    std::set<std::vector<int>> seen;
    std::vector<std::vector<int>> todo{{}};
    while (!todo.empty()) {
        const std::vector<int> prefix = todo.back();
        todo.pop_back();
        for (int i = 0; i < N; ++i) mem[i].v = start[i];
        for (int t = 0; t < kThreads; ++t) {
            Fiber& f = fibers[t];
            f.reads.clear();
            f.done = false;
            getcontext(&f.ctx);
            f.ctx.uc_stack.ss_sp = f.stack.data();
            f.ctx.uc_stack.ss_size = f.stack.size();
            f.ctx.uc_link = nullptr;
            makecontext(&f.ctx, entry, 0);
            turn(t, true);  // up to its first step
        }
        std::vector<int> taken(kThreads, 0);
        for (int t : prefix) {
            turn(t);
            ++taken[t];
        }
        std::vector<int> state;
        for (int i = 0; i < N; ++i) state.push_back(mem[i].v);
        const Mem now = state;
        bool alive = false;
        for (int t = 0; t < kThreads; ++t) {
            state.push_back(-taken[t] - 1);
            state.insert(state.end(), fibers[t].reads.begin(), fibers[t].reads.end());
            alive |= !fibers[t].done;
        }
        if (!seen.insert(state).second) continue;
        if (!alive) {
            out.insert(now);
            continue;
        }
        for (int t = 0; t < kThreads; ++t)
            if (!fibers[t].done) {
                todo.push_back(prefix);
                todo.back().push_back(t);
            }
    }
    return out;
}

// Compression of every forest on a path of the points (each parent smaller or
// the point itself): every point of three has to end at its root.
static int compress() {
    long cases = 0;
    for (int f = 0; f < 2 * 3 * 4 * 5; ++f) {
        const Mem start{0, f % 2, f / 2 % 3, f / 6 % 4, f / 24, 5};
        for (int skip = 0; skip < 5; ++skip) {  // three of points 1 to 4, or the last three
            std::vector<int> points;
            for (int i = 1; i < 5; ++i)
                if (i != skip && (skip || i > 1)) points.push_back(i);
            ++cases;
            body = [&](int t) { compress_point(mem, points[t]); };
            for (const Mem& end : outcomes(start))
                for (int p : points) {
                    int root = p;
                    while (start[root] != root) root = start[root];
                    if (end[p] == root) continue;
                    std::printf("not at its root: %d of", p);
                    for (int v : start) std::printf(" %d", v);
                    std::printf(", at the end");
                    for (int v : end) std::printf(" %d", v);
                    std::printf("\n");
                    return 1;
                }
        }
    }
    std::printf("%ld cases\n", cases);
    return 0;
}

int main(int argc, char** argv) {
    if (argc == 2) return compress();
    if (argc != 3) return 2;
    const int n = std::atoi(argv[1]);
    const bool carried = std::atoi(argv[2]) != 0;
    long cases = 0, ends = 0;
    for (int old = 0; old < 64; ++old) {  // the old set's three members, its smallest their root
        if (__builtin_popcount((unsigned)old) != 3) continue;
        std::vector<int> members, fresh;
        for (int i = 0; i < N; ++i) (old >> i & 1 ? members : fresh).push_back(i);
        Mem start(N);
        for (int i = 0; i < N; ++i) start[i] = i;
        for (int q : members) start[q] = members[0];
        for (int e = 0; e < 27; ++e) {  // every new point's edge: to one of the old members
            const int to[3] = {members[e % 3], members[e / 3 % 3], members[e / 9]};
            ++cases;
            body = [&](int t) {  // k_hook
                RootSpan span(round_root(mem, fresh[t], n, carried));
                span.see(round_root(mem, to[t], n, carried));
                span.hook(mem);
            };
            for (const Mem& hooked : outcomes(start)) {
                ++ends;
                for (int i = 0; i < N; ++i) mem[i].v = hooked[i];
                for (int t = 0; t < kThreads; ++t) unite(mem, fresh[t], to[t]);  // k_union_tiles, new edges
                for (int i = 0; i < N; ++i) {
                    if (find_root(mem, i) == find_root(mem, 0)) continue;
                    std::printf("split: old members %d %d %d, new points %d-%d %d-%d %d-%d, after hooking", members[0],
                                members[1], members[2], fresh[0], to[0], fresh[1], to[1], fresh[2], to[2]);
                    for (int v : hooked) std::printf(" %d", v);
                    std::printf("\n");
                    return 1;
                }
            }
        }
    }
    std::printf("%ld cases, %ld outcomes of the hooking\n", cases, ends);
    return 0;
}

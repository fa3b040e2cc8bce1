// Maximal k-biplex search of small graphs on bit masks (sm_100a device code).
//
// A graph with at most 32 N vertices on each side (N = 1 to 4) fits a warp's
// registers: lane i holds U vertices i, i + 32, ... and V vertices i, i + 32,
// ..., each as the mask of the vertices of the other side that it misses.  A
// search state is four masks, the same in all lanes: the included (I) and the
// undecided (C) vertices of each side; every other vertex is excluded, so a
// state describes its subproblem completely.  A node is a few popcounts and
// ballots, with no list, no frame and no adjacency probe:
//   misses of v in I u C     popc(miss mask & (I | C) of the other side)
//   pruned                   an excluded vertex with at most k misses that
//                            misses no vertex with k or more can join every
//                            leaf below
//   result                   no vertex of I u C has more than k misses (and
//                            nothing can join)
//   forced                   candidates with at most k misses that miss no
//                            vertex with more than k are in every maximal leaf
//   at most 5 candidates     every subset of them is tested, one per lane
//   branch                   take the included vertex v with the most misses
//                            (over k; at most k of them can stay), and of the
//                            candidates it misses the one with the most misses:
//                            it is included, or it is excluded
//   fan                      when v has one miss left, at most one of the
//                            candidates P it misses can be included: one child
//                            per w in P (the rest of P is out, v has k misses
//                            then) and the state without P
// Root task: x in U with I = {x}, C = the U vertices after x and all V
// vertices, or, for a range of first-level children y, one state (x, y) after
// the other (C: after x, after y).
//
// States waiting on the warp's stack are handed to idle warps (tickets and
// slots, as in the list-based kernel; a record is one stack entry, and its slot
// holds it, so there is no separate index).  Slots are used again (state_ring.h):
// a search of any length stays shared to its end.
//
// What bounds it: integer issue, and on graphs of a few thousand nodes the
// latency of one warp's chain of nodes.  The list-based search of the same
// graphs spent 1 000-1 600 warp instructions a node on hash probes, frames and
// lists, and their L2 latency; this one spent 640 with N = 3 masks (77 x 77, k
// = 2, before the fans: 10.3 G instructions for 12.4 M results, 43 % of the
// issue slots active) and nothing leaves the SM.  Measured, complete runs, list-based -> here (ms,
// one B200): 18 x 14 k = 1 0.90 -> 0.12, k = 3 19.5 -> 0.29; 58 x 58 k = 2 30.3 ->
// 2.4; 77 x 77 k = 2 115 -> 10.6; 82 x 83 k = 2 31.6 -> 8.5; 128 x 128 k = 1
// 10.4 -> 2.2.
#pragma once
#include "enum_warp.cuh"
#include "state_ring.h"

namespace gmk {
namespace dense {

using warp::kFull;
using warp::bcast;
using warp::lanemask_lt;

constexpr uint32_t kSubset = 5;        // 2^5 subsets: one per lane
constexpr uint32_t kMinShare = 10;     // candidates of a state worth handing on (7: up to 10 %
                                       //   slower on 18 x 14 graphs, 14: 1.8x at k = 3)
// Nodes between two looks at the shared counters.  N = 1: 8 ran a 18 x 14 graph
// 1.3x faster than 4 at k = 1 (16: 1.35x, but 1.4x slower at k = 3); with more
// mask words a node costs more, and 4 is 5-10 % faster than 2 or 8.
template <int N> __host__ __device__ constexpr uint32_t poll_nodes() { return N == 1 ? 8 : 4; }
// A record: mark (written last), graph, 2 spare words, a state.  All N use one
// record size: a record is recognised by the mark in its first word, which must
// never have been another launch's state word.
constexpr uint32_t kHeader = 4;
constexpr unsigned long long kRingLimitNs = 10000000000ull;   // a slot not read for 10 s: an error
constexpr uint32_t kRecordWords = kHeader + 21;
// Stack entries in shared memory; deeper ones are in the warp's global spill
// area.  One entry per included candidate on the path (a fan leaves one for all
// its children, and each has fewer candidates).
template <int N> __host__ __device__ constexpr uint32_t shared_depth() { return N == 1 ? 64 : N == 2 ? 32 : 16; }
// Fans (the children that include one of P each, and the state without P, in
// place of a chain of include / exclude states) where P has 6 vertices or more:
// the chain's exclude states are nodes that decide nothing, -41 % nodes at 60 x
// 60, 180 edges, k = 2: 2.98 to 2.35 ms; 80 x 80, 320 edges, k = 2: 14.3 to
// 10.6; 50 x 50, 120 edges, k = 3: 174 to 125; 128 x 128, 1200 edges, k = 1: 2.79
// to 2.19.  From 4 on: 2.06 at the last, but 0.51 in place of 0.47 ms at 60 x
// 60, 300 edges, k = 1; from 8 on: 2.4 and 0.47.  With one word a side the run is
// a chain of few states and a fan is handed on as a whole: 30 x 30, 155 edges, k =
// 1 takes 0.23 ms with fans and 0.17 without.
template <int N> constexpr bool kFans = N > 1;
constexpr uint32_t kFanMin = 6;
// An entry: a state, and the children of a fan that are still to be searched
// before it (their mask, and its side: 0 none, 1 U, 2 V).
template <int N> __host__ __device__ constexpr uint32_t entry_words() { return kFans<N> ? 5 * N + 1 : 4 * N; }
template <int N> __host__ __device__ constexpr uint32_t spill_words() {
    return (64 * N - shared_depth<N>()) * entry_words<N>();
}

template <int N>
struct State {
    uint32_t iu[N], iv[N], cu[N], cv[N];
};

template <int N>
struct Shared {
    uint32_t stack[shared_depth<N>()][entry_words<N>()];
    uint32_t found[64][2 * N];                     // results not yet hashed: U and V masks
    unsigned long long ea[64 * N], eb[64 * N];     // hash elements (U at 0, V at 32 N)
};

struct Share {
    uint32_t* rec;                    // fixed-size records, one per slot of the ring
    StateRing ring;
    unsigned long long* tail;         // tickets reserved
    unsigned long long* claim;        // tickets taken by waiting warps
    unsigned long long* outstanding;  // unfinished tasks - queue_len (mod 2^64)
    unsigned long long* donated;
    int* done;                        // warp::kDoneFlags flags, as warp::Donation's
    int* stop;                        // the launch's stop and error words
    int* error;
    uint32_t min_nodes;
};

template <int N>
struct Ctx {
    uint32_t nu, nv, k, lane;
    uint32_t um[N][N], vm[N][N];      // [i]: this lane's vertex 32 i + lane; the vertices it misses
    Shared<N>* sh;
    uint32_t* spill;
    uint32_t nfound, sp, bottom;      // stack entries [bottom, sp)
    uint32_t extra;                   // nodes that subset tests of this task stood for
    unsigned long long cnt, hsum, hxor, nodes, work;
};

// Bits 0..n-1 of word w of an N-word mask.
__device__ __forceinline__ uint32_t low_bits(uint32_t n, uint32_t w) {
    return n >= 32 * w + 32 ? kFull : n > 32 * w ? (1u << (n - 32 * w)) - 1u : 0u;
}

template <int N>
__device__ __forceinline__ uint32_t misses(const uint32_t (&m)[N], const uint32_t (&x)[N]) {
    uint32_t c = 0;
    #pragma unroll
    for (int w = 0; w < N; ++w) c += __popc(m[w] & x[w]);
    return c;
}
template <int N>
__device__ __forceinline__ bool meets(const uint32_t (&m)[N], const uint32_t (&x)[N]) {
    uint32_t a = 0;
    #pragma unroll
    for (int w = 0; w < N; ++w) a |= m[w] & x[w];
    return a != 0;
}

// The graph's miss masks and hash elements.
template <int N>
__device__ __forceinline__ void load_graph(Ctx<N>& t, const GraphView& g) {
    t.nu = g.nl;
    t.nv = g.n - g.nl;
    #pragma unroll
    for (int i = 0; i < N; ++i) {
        #pragma unroll
        for (int w = 0; w < N; ++w) { t.um[i][w] = low_bits(t.nv, w); t.vm[i][w] = low_bits(t.nu, w); }
        const uint32_t v = 32u * i + t.lane;
        if (v < t.nu) {
            const uint32_t a = g.off[v], b = g.off[v + 1];
            t.work += b - a;
            #pragma unroll 4
            for (uint32_t p = a; p < b; ++p) {
                const uint32_t y = g.adj[p] - g.nl;
                #pragma unroll
                for (int w = 0; w < N; ++w) t.um[i][w] &= y >> 5 == (uint32_t)w ? ~(1u << (y & 31u)) : kFull;
            }
        }
        if (v < t.nv) {
            const uint32_t a = g.off[g.nl + v], b = g.off[g.nl + v + 1];
            t.work += b - a;
            #pragma unroll 4
            for (uint32_t p = a; p < b; ++p) {
                const uint32_t x = g.adj[p];
                #pragma unroll
                for (int w = 0; w < N; ++w) t.vm[i][w] &= x >> 5 == (uint32_t)w ? ~(1u << (x & 31u)) : kFull;
            }
        }
        const unsigned long long eu = elem_a(v), ev = elem_a(g.nl + v);
        t.sh->ea[v] = eu;
        t.sh->eb[v] = elem_b(eu);
        t.sh->ea[32 * N + v] = ev;
        t.sh->eb[32 * N + v] = elem_b(ev);
    }
    __syncwarp();
}

// Hashes the buffered results, one per lane.
template <int N>
__device__ __forceinline__ void flush_found(Ctx<N>& t) {
    __syncwarp();
    #pragma unroll 1
    for (uint32_t base = 0; base < t.nfound; base += 32) {
        unsigned long long h1 = 0, h2 = 0;
        if (base + t.lane < t.nfound) {
            unsigned long long x = 0, y = 0;
            uint32_t nx = 0, ny = 0;
            #pragma unroll 1
            for (int w = 0; w < 2 * N; ++w) {
                const uint32_t f = t.sh->found[base + t.lane][w];
                if (w < N) nx += __popc(f); else ny += __popc(f);
                #pragma unroll 1
                for (uint32_t m = f; m; m &= m - 1) {
                    const uint32_t e = 32 * w + __ffs(m) - 1;
                    x += t.sh->ea[e];
                    y += t.sh->eb[e];
                }
            }
            h1 = final_h1(x, nx, ny);
            h2 = final_h2(y, nx, ny);
        }
        t.hsum += warp::warp_sum64(h1);
        t.hxor ^= ((unsigned long long)__reduce_xor_sync(kFull, (uint32_t)(h2 >> 32)) << 32) |
                  __reduce_xor_sync(kFull, (uint32_t)h2);
    }
    t.cnt += t.nfound;
    t.nfound = 0;
    __syncwarp();
}

// Drops the candidates that no longer fit I: more than k misses in I, or a
// missed vertex of I that has k already.
template <int N>
__device__ __forceinline__ void refit(const Ctx<N>& t, State<N>& s) {
    const uint32_t k = t.k, lane = t.lane;
    uint32_t xu[N], xv[N], su[N], sv[N];
    #pragma unroll
    for (int i = 0; i < N; ++i) { xu[i] = misses<N>(t.um[i], s.iv); xv[i] = misses<N>(t.vm[i], s.iu); }
    #pragma unroll
    for (int i = 0; i < N; ++i) {
        su[i] = __ballot_sync(kFull, ((s.iu[i] >> lane) & 1u) && xu[i] >= k);
        sv[i] = __ballot_sync(kFull, ((s.iv[i] >> lane) & 1u) && xv[i] >= k);
    }
    #pragma unroll
    for (int i = 0; i < N; ++i) {
        s.cu[i] &= __ballot_sync(kFull, xu[i] <= k && !meets<N>(t.um[i], sv));
        s.cv[i] &= __ballot_sync(kFull, xv[i] <= k && !meets<N>(t.vm[i], su));
    }
}

// Subsets T of C, one per lane: is I u T (masks lu, lv) a result?  *feasible: how
// many of them are k-biplexes -- the nodes of their set-enumeration tree, which
// this one node stands for.
template <int N>
__device__ __forceinline__ bool subsets(const Ctx<N>& t, const State<N>& s, uint32_t (&lu)[N],
                                        uint32_t (&lv)[N], uint32_t* feasible) {
    const uint32_t lane = t.lane, k = t.k;
    uint32_t j = 0, any_v = 0;
    uint32_t hu[N], hv[N];
    #pragma unroll
    for (int w = 0; w < N; ++w) {
        lu[w] = s.iu[w];
        hu[w] = hv[w] = 0;
        #pragma unroll 1
        for (uint32_t y = s.cu[w]; y; y &= y - 1, ++j) lu[w] |= ((lane >> j) & 1u) ? (y & (0u - y)) : 0u;
    }
    #pragma unroll
    for (int w = 0; w < N; ++w) {
        lv[w] = s.iv[w];
        #pragma unroll 1
        for (uint32_t y = s.cv[w]; y; y &= y - 1, ++j) lv[w] |= ((lane >> j) & 1u) ? (y & (0u - y)) : 0u;
        any_v |= lv[w];
    }
    bool alive = (lane >> j) == 0;
    // members: misses, blockers (k or more)
    #pragma unroll
    for (int w = 0; w < N; ++w) {
        #pragma unroll 1
        for (uint32_t y = s.iu[w] | s.cu[w]; y; y &= y - 1) {
            const uint32_t i = __ffs(y) - 1;
            uint32_t c = 0;
            #pragma unroll
            for (int q = 0; q < N; ++q) c += __popc(__shfl_sync(kFull, t.um[w][q], i) & lv[q]);
            if ((lu[w] >> i) & 1u) {
                alive = alive && c <= k;
                hu[w] |= c >= k ? 1u << i : 0u;
            }
        }
        #pragma unroll 1
        for (uint32_t y = s.iv[w] | s.cv[w]; y; y &= y - 1) {
            const uint32_t i = __ffs(y) - 1;
            uint32_t c = 0;
            #pragma unroll
            for (int q = 0; q < N; ++q) c += __popc(__shfl_sync(kFull, t.vm[w][q], i) & lu[q]);
            if ((lv[w] >> i) & 1u) {
                alive = alive && c <= k;
                hv[w] |= c >= k ? 1u << i : 0u;
            }
        }
    }
    *feasible = __popc(__ballot_sync(kFull, alive));
    alive = alive && any_v != 0;
    // nothing left out may join.  A vertex that misses more than k of I, or a
    // vertex of I with k misses in I, joins none of the subsets: only the
    // others are tested subset by subset.
    State<N> other;
    #pragma unroll
    for (int w = 0; w < N; ++w) {
        other.iu[w] = s.iu[w]; other.iv[w] = s.iv[w];
        other.cu[w] = low_bits(t.nu, w) & ~s.iu[w];
        other.cv[w] = low_bits(t.nv, w) & ~s.iv[w];
    }
    refit<N>(t, other);
    #pragma unroll
    for (int w = 0; w < N; ++w) {
        #pragma unroll 1
        for (uint32_t y = other.cu[w]; y; y &= y - 1) {
            const uint32_t i = __ffs(y) - 1;
            uint32_t c = 0, b = 0;
            #pragma unroll
            for (int q = 0; q < N; ++q) {
                const uint32_t m = __shfl_sync(kFull, t.um[w][q], i);
                c += __popc(m & lv[q]);
                b |= m & hv[q];
            }
            if (!((lu[w] >> i) & 1u) && c <= k && !b) alive = false;
        }
        #pragma unroll 1
        for (uint32_t y = other.cv[w]; y; y &= y - 1) {
            const uint32_t i = __ffs(y) - 1;
            uint32_t c = 0, b = 0;
            #pragma unroll
            for (int q = 0; q < N; ++q) {
                const uint32_t m = __shfl_sync(kFull, t.vm[w][q], i);
                c += __popc(m & lu[q]);
                b |= m & hu[q];
            }
            if (!((lv[w] >> i) & 1u) && c <= k && !b) alive = false;
        }
    }
    return alive;
}

template <int N>
__device__ __forceinline__ uint32_t* stack_at(const Ctx<N>& t, uint32_t i) {
    return i < shared_depth<N>() ? t.sh->stack[i] : t.spill + (i - shared_depth<N>()) * entry_words<N>();
}
template <int N>
__device__ __forceinline__ void push(Ctx<N>& t, const State<N>& s, const uint32_t (&p)[N], uint32_t side) {
    uint32_t* e = stack_at<N>(t, t.sp);
    if (t.lane == 0) {
        #pragma unroll
        for (int w = 0; w < N; ++w) {
            e[w] = s.iu[w]; e[N + w] = s.iv[w]; e[2 * N + w] = s.cu[w]; e[3 * N + w] = s.cv[w];
            if (kFans<N> && side) e[4 * N + w] = p[w];
        }
        if (kFans<N>) e[5 * N] = side;
    }
    ++t.sp;
}
template <int N>
__device__ __forceinline__ void read_state(const uint32_t* e, State<N>& s) {
    #pragma unroll
    for (int w = 0; w < N; ++w) {
        s.iu[w] = e[w]; s.iv[w] = e[N + w]; s.cu[w] = e[2 * N + w]; s.cv[w] = e[3 * N + w];
    }
}

// The next waiting state: the top entry's first remaining child (true: to be
// refitted), else its state.
template <int N>
__device__ __forceinline__ bool pop(Ctx<N>& t, State<N>& s) {
    if (!kFans<N>) {
        --t.sp;
        __syncwarp();
        read_state<N>(stack_at<N>(t, t.sp), s);
        __syncwarp();
        return false;
    }
    __syncwarp();
    uint32_t* e = stack_at<N>(t, t.sp - 1);
    read_state<N>(e, s);
    const uint32_t side = e[5 * N];
    if (side == 0) {
        --t.sp;
        __syncwarp();
        return false;
    }
    uint32_t bit = 0, left = 0;
    int word = 0;
    #pragma unroll
    for (int w = N - 1; w >= 0; --w) {
        const uint32_t p = e[4 * N + w];
        left = p ? left | bit | (p & (p - 1)) : left;
        if (p) { word = w; bit = p & (0u - p); }
    }
    #pragma unroll
    for (int w = 0; w < N; ++w) {
        const uint32_t m = word == w ? bit : 0u;
        if (side == 1) s.iu[w] |= m; else s.iv[w] |= m;
    }
    __syncwarp();
    if (t.lane == 0) {
        e[4 * N + word] &= ~bit;
        if (!left) e[5 * N] = 0;
    }
    return true;
}

// One node: prunes, takes results, or goes on (true) to the child that includes the
// branching candidate, to be refitted; the state that excludes it is pushed.  A fan is
// pushed as one entry (false): pop hands out its children, to be refitted too, and
// then the state without them.
template <int N>
__device__ __forceinline__ bool node(Ctx<N>& t, State<N>& s, bool fit) {
    if (kFans<N> && fit) refit<N>(t, s);
    const uint32_t lane = t.lane, k = t.k;
    uint32_t lu[N], lv[N], tu[N], tv[N], hu[N], hv[N], bu[N], bv[N];
    uint32_t any_v = 0, any_b = 0;
    #pragma unroll
    for (int w = 0; w < N; ++w) { lu[w] = s.iu[w] | s.cu[w]; lv[w] = s.iv[w] | s.cv[w]; any_v |= lv[w]; }
    if (!any_v) return false;
    #pragma unroll
    for (int i = 0; i < N; ++i) { tu[i] = misses<N>(t.um[i], lv); tv[i] = misses<N>(t.vm[i], lu); }
    #pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool inu = (lu[i] >> lane) & 1u, inv = (lv[i] >> lane) & 1u;
        hu[i] = __ballot_sync(kFull, inu && tu[i] >= k);
        hv[i] = __ballot_sync(kFull, inv && tv[i] >= k);
        bu[i] = __ballot_sync(kFull, inu && tu[i] > k);
        bv[i] = __ballot_sync(kFull, inv && tv[i] > k);
        any_b |= bu[i] | bv[i];
    }
    bool add = false;
    #pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t v = 32u * i + lane;
        add |= v < t.nu && !((lu[i] >> lane) & 1u) && tu[i] <= k && !meets<N>(t.um[i], hv);
        add |= v < t.nv && !((lv[i] >> lane) & 1u) && tv[i] <= k && !meets<N>(t.vm[i], hu);
    }
    if (__any_sync(kFull, add)) return false;
    bool hit = lane == 0;
    if (any_b) {
        uint32_t left = 0;
        #pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t fu = __ballot_sync(kFull, ((s.cu[i] >> lane) & 1u) && tu[i] <= k && !meets<N>(t.um[i], bv));
            const uint32_t fv = __ballot_sync(kFull, ((s.cv[i] >> lane) & 1u) && tv[i] <= k && !meets<N>(t.vm[i], bu));
            s.iu[i] |= fu; s.cu[i] &= ~fu;
            s.iv[i] |= fv; s.cv[i] &= ~fv;
            left += __popc(s.cu[i]) + __popc(s.cv[i]);
        }
        if (left > kSubset) {
            // the worst included vertex (key: misses, then position from the top)
            uint32_t best = 0;
            #pragma unroll
            for (int i = 0; i < N; ++i) {
                const uint32_t a = (((s.iu[i] & bu[i]) >> lane) & 1u) ? (tu[i] << 8 | (255u - (32 * i + lane))) : 0u;
                const uint32_t b = (((s.iv[i] & bv[i]) >> lane) & 1u) ? (tv[i] << 8 | (127u - (32 * i + lane))) : 0u;
                best = a > best ? a : best;
                best = b > best ? b : best;
            }
            best = __reduce_max_sync(kFull, best);
            uint32_t pu[N], pv[N];
            #pragma unroll
            for (int w = 0; w < N; ++w) { pu[w] = s.cu[w]; pv[w] = s.cv[w]; }
            if (best) {
                const uint32_t at = 255u - (best & 255u);   // U at 0, V at 128
                const bool on_u = at < 128;
                uint32_t cur = 0, np = 0;
                #pragma unroll
                for (int w = 0; w < N; ++w) {
                    uint32_t mu = 0, mv = 0;
                    #pragma unroll
                    for (int i = 0; i < N; ++i) {
                        if (((at & 127u) >> 5) == (uint32_t)i) { mu = t.um[i][w]; mv = t.vm[i][w]; }
                    }
                    const uint32_t m = __shfl_sync(kFull, on_u ? mu : mv, at & 31u);
                    pu[w] &= on_u ? 0u : m;
                    pv[w] &= on_u ? m : 0u;
                    cur += __popc(m & (on_u ? s.iv[w] : s.iu[w]));
                    np += __popc(pu[w] | pv[w]);
                }
                if (kFans<N> && cur + 1 == k && np >= kFanMin) {
                    // a fan: at most one of p
                    uint32_t p[N];
                    #pragma unroll
                    for (int w = 0; w < N; ++w) {
                        p[w] = on_u ? pv[w] : pu[w];
                        s.cu[w] &= ~pu[w];
                        s.cv[w] &= ~pv[w];
                    }
                    push<N>(t, s, p, on_u ? 2u : 1u);
                    return false;
                }
            }
            best = 0;
            #pragma unroll
            for (int i = 0; i < N; ++i) {
                const uint32_t a = ((pu[i] >> lane) & 1u) ? (tu[i] << 8 | (255u - (32 * i + lane))) : 0u;
                const uint32_t b = ((pv[i] >> lane) & 1u) ? (tv[i] << 8 | (127u - (32 * i + lane))) : 0u;
                best = a > best ? a : best;
                best = b > best ? b : best;
            }
            const uint32_t at = 255u - (__reduce_max_sync(kFull, best) & 255u);
            const uint32_t bit = 1u << (at & 31u), word = (at & 127u) >> 5;
            #pragma unroll
            for (int w = 0; w < N; ++w) {
                const uint32_t m = word == (uint32_t)w ? bit : 0u;
                if (at < 128) s.cu[w] &= ~m; else s.cv[w] &= ~m;
            }
            push<N>(t, s, pu, 0u);
            #pragma unroll
            for (int w = 0; w < N; ++w) {
                const uint32_t m = word == (uint32_t)w ? bit : 0u;
                if (at < 128) s.iu[w] |= m; else s.iv[w] |= m;
            }
            if (!kFans<N>) refit<N>(t, s);
            return true;
        }
        uint32_t feasible;
        hit = subsets<N>(t, s, lu, lv, &feasible);
        t.extra += feasible - 1;
    }
    const uint32_t who = __ballot_sync(kFull, hit);
    if (hit) {
        uint32_t* f = t.sh->found[t.nfound + __popc(who & lanemask_lt())];
        #pragma unroll
        for (int w = 0; w < N; ++w) { f[w] = lu[w]; f[N + w] = lv[w]; }
    }
    t.nfound += __popc(who);
    if (t.nfound > 32) flush_found<N>(t);
    return false;
}

// Tickets that wait for a record (lane 0), at most 32; kWantChecked in it: they
// are to be counted again (waiting_now) before any is served.
constexpr uint32_t kWantChecked = 64;
__device__ __forceinline__ uint32_t waiting(const Share& sh) {
    const unsigned long long tail = *(volatile const unsigned long long*)sh.tail;
    const long long w = (long long)(*(volatile const unsigned long long*)sh.claim - tail);
    return w <= 0 ? 0u : (uint32_t)(w < 32 ? w : 32) | (sh.ring.early(tail) ? 0u : kWantChecked);
}
// The same as of one moment: the claimed tickets are read before the reserved ones.
__device__ __forceinline__ uint32_t waiting_now(const Share& sh) {
    unsigned long long claim;
    asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(claim) : "l"(sh.claim) : "memory");
    const long long w = (long long)(claim - *(volatile const unsigned long long*)sh.tail);
    return w > 0 ? (uint32_t)(w < 32 ? w : 32) : 0u;
}

// Waits until the slot r of `ticket` has been read by its last user (a warp that
// runs: one look, as a rule).  False: the launch stops, or the wait ran out.
__device__ __forceinline__ bool ring_wait(const Share& sh, unsigned long long ticket, const uint32_t* r) {
    if (sh.ring.first(ticket)) return true;
    unsigned long long since = 0;
    #pragma unroll 1
    for (uint32_t spin = 0; !sh.ring.free(ticket, *(volatile const uint32_t*)r); ++spin) {
        if (load_flag(sh.stop)) return false;
        const unsigned long long now = now_ns();
        if (spin == 0) since = now;
        if (now - since > kRingLimitNs) {
            atomicCAS(sh.error, 0, TASK_E_TIMEOUT);
            atomicExch(sh.stop, 1);
            return false;
        }
        __nanosleep(64);
    }
    return true;       // (the caller's stores wait for the branch)
}

// Hands up to `want` of the oldest entries (those with kMinShare candidates
// and children or more) to waiting warps.
template <int N>
__device__ __forceinline__ void donate(Ctx<N>& t, const Share& sh, uint32_t gid, uint32_t want) {
    __syncwarp();
    const bool checked = want & kWantChecked;
    want &= kWantChecked - 1;
    uint32_t n = t.sp - t.bottom;
    n = n < want ? n : want;
    n = n < kRingShare ? n : kRingShare;
    // lane i < n: the i-th oldest; the run of large ones from the bottom
    uint32_t c = 0;
    if (t.lane < n) {
        const uint32_t* e = stack_at<N>(t, t.bottom + t.lane);
        #pragma unroll
        for (int w = 2 * N; w < 4 * N; ++w) c += __popc(e[w]);
        if (kFans<N> && e[5 * N]) {
            #pragma unroll
            for (int w = 4 * N; w < 5 * N; ++w) c += __popc(e[w]);
        }
    }
    const uint32_t small = __ballot_sync(kFull, t.lane >= n || c < kMinShare);
    n = __ffs(small) - 1;      // (n <= kRingShare < 32: some lane is set)
    if (n == 0) return;
    if (checked) {
        want = bcast(waiting_now(sh));
        n = n < want ? n : want;
        if (n == 0) return;
    }
    unsigned long long ticket = 0;
    if (t.lane == 0) {
        ticket = atomicAdd(sh.tail, (unsigned long long)n);
        atomicAdd(sh.outstanding, (unsigned long long)n);   // before they can finish
        atomicAdd(sh.donated, (unsigned long long)n);
    }
    ticket = bcast(ticket) + t.lane;
    if (t.lane < n) {
        uint32_t* r = sh.rec + (unsigned long long)sh.ring.slot(ticket) * kRecordWords;
        if (ring_wait(sh, ticket, r)) {
            const uint32_t* e = stack_at<N>(t, t.bottom + t.lane);
            r[1] = gid;
            #pragma unroll
            for (uint32_t w = 0; w < entry_words<N>(); ++w) r[kHeader + w] = e[w];
            __threadfence();
            atomicExch(r, sh.ring.ready(ticket));
        }
    }
    __syncwarp();
    t.bottom += n;
    __syncwarp();
}

}  // namespace dense
}  // namespace gmk

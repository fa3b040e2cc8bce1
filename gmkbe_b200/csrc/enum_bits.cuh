// Bit-mask search of a node whose candidates are few (sm_100a device code).
//
// A node (S, C) with both candidate sides local and at most 32 U and 32 V
// vertices in S u C is searched on bit masks, without frames, lists or hash
// probes.  Lane i holds U vertex i and V vertex i of the node's universe
// (members first, then candidates, in list order) with one 32-bit mask each:
// the vertices of the other side it misses.  A state of the search is four
// warp-uniform masks, the included (I) and undecided (C) vertices per side,
// and the test of a whole node is a few popcounts and ballots:
//   misses of v in S u C        popc(miss mask & (I | C) of the other side)
//   blockers                    ballot(misses >= k)
//   addable outsider            an excluded universe vertex (its lane) or an
//                               outside vertex (one mask each, kept by lane)
//                               with at most k misses and no missed blocker
//   forced candidates           all at once: misses <= k, no missed violator
// The rules are those of enter_node; the branching differs: the candidate
// with the most misses is taken in, and left out (a left-out candidate joins
// the outsiders at once, so a branch that it fills is cut there): among those that
// the worst violator in I misses, when there is one (1.2-1.8 times fewer nodes
// than taking the worst candidate of all).  Nodes with
// at most kBitsSubset candidates test all subsets, one per lane.
//
// Outside vertices.  A vertex of side s that can join some leaf below misses
// at most k members of S_o and no member at k misses, so it lies in the row of
// a saturated member, or in one of any k + 1 members' rows.  Those rows are
// scanned once per universe.
//
// What bounds it: instruction fetch and latency (er200 k = 1: 3.3 G warp
// instructions for 1.83 M results, most of them setting universes up).  A node of
// the list-based search costs 1 000-1 600 warp instructions, hash probes and list
// traffic, one on masks 100-400.  Measured with lane blocks and the wider
// register allocation (ms, complete runs, one B200): er200 k = 1 27.6 -> 11.5, 400 x
// 400 degree 5 19.7 -> 6.6, 200 x 200 degree 5, k = 2, first 3 10^6 28.0 -> 6.9.
#pragma once

namespace gmk {
namespace warp {

constexpr uint32_t kBitsSide = 32;       // universe vertices per side: one per lane
constexpr uint32_t kBitsScanMax = 2048;  // a lane block child: entries of the row that bounds the other side
// Entries of the rows that bound one side's outsiders at a node that the list-based
// search hands over.  Below a hub they number hundreds, each with its probes, for
// subtrees of a node or two, where the list-based rules stop at the first vertex that
// can join: 168 x 39 with hubs of 168, k = 1, counted without sharing 6.0 ms with rows
// up to 2 048, 4.6 with 160 (and with 64); er200 and the Chung-Lu prefixes have shorter
// ones.
constexpr uint32_t kBitsRow = 160;
constexpr uint32_t kBitsSubset = 5;   // 2^5 subsets: one per lane
constexpr uint32_t kBitsStack = 64;      // one entry per included candidate, at most
constexpr uint32_t kBitsBudget = 8;   // nodes between two polls of the search loop

// Shared memory of one warp's bit search.
struct BitShared {
    uint4 stack[kBitsStack];             // left-out states to come back to: IU, IV, CU, CV
    unsigned long long ea[64], eb[64];   // hash elements of the universe (U at 0, V at 32)
    uint2 found[64];                     // results not yet hashed: their U and V masks
    uint32_t ids[64];                    // the universe's ids
};

// Rows to scan for the outside vertices: lane i holds source i (row offset,
// first entry of the joint scan, side of its outsiders << 5 | universe index).
struct BitSources {
    uint32_t row, start, info;
    uint32_t n, total;
};

struct Bits {
    bool active;
    bool lanes;                     // the node is a child that lane_blocks found
    bool hashed;                    // ea / eb are filled
    uint32_t iu, iv, cu, cv;        // the state to look at next (uniform)
    uint32_t su, sv;                // members with k misses in S (set-up only)
    uint32_t um, vm;                // this lane's U / V vertex: the vertices it misses
    uint32_t ou, ov;                // this lane's outside U / V vertex (first 32)
    uint32_t nu, nv;                // universe sizes
    uint32_t nou, nov;              // outside vertices of U / V
    uint32_t over;                  // arena offset of the outside vertices past 32 per side
    uint32_t sp, bottom;            // stack entries [bottom, sp)
    uint32_t nfound;
    BitShared* sh;
};

// Outside vertex r >= 32 of U / V (V vertices from the end of the region).
__device__ __forceinline__ uint32_t bits_over_u(const Ctx& t, const Bits& b, uint32_t r) {
    return t.arena[b.over + (r - 32)];
}
__device__ __forceinline__ uint32_t bits_over_v(const Ctx& t, const Bits& b, uint32_t r) {
    return t.arena[t.cap - 1 - (r - 32)];
}

__device__ __forceinline__ unsigned long long warp_xor64(unsigned long long v) {
    return ((unsigned long long)__reduce_xor_sync(kFull, (uint32_t)(v >> 32)) << 32) |
           __reduce_xor_sync(kFull, (uint32_t)v);
}

// Adds the rows that hold side s's outsiders: that of the saturated member
// (universe mask `sat`) with the lowest degree, or the k + 1 lowest-degree rows
// among the members `mem` of the other side, whichever is shorter.  d, r:
// degree and row offset of this lane's vertex of that side.  False: neither
// exists, or the rows are too long.
__device__ __forceinline__ bool bits_source(const Ctx& t, BitSources& src, int s, uint32_t mem,
                                            uint32_t sat, uint32_t d, uint32_t r) {
    const uint32_t lane = t.lane, k = t.k;
    const uint32_t key = d < (1u << 26) ? d << 5 | lane : kFull - 31 + lane;
    uint32_t pick = 0, cost = kFull;
    if (sat) {
        const uint32_t best = __reduce_min_sync(kFull, ((sat >> lane) & 1u) ? key : kFull);
        pick = 1u << (best & 31u);
        cost = best >> 5;
    }
    if (cost > 32 && (uint32_t)__popc(mem) > k) {
        uint32_t left = mem, sum = 0, pk = 0;
        #pragma unroll 1
        for (uint32_t c = 0; c <= k; ++c) {
            const uint32_t best = __reduce_min_sync(kFull, ((left >> lane) & 1u) ? key : kFull);
            const uint32_t bit = 1u << (best & 31u);
            left &= ~bit;
            pk |= bit;
            sum += best >> 5;   // (k + 1 <= 16 terms below 2^27)
        }
        if (sum < cost) { pick = pk; cost = sum; }
    }
    if (cost > kBitsRow) return false;
    #pragma unroll 1
    for (; pick; pick &= pick - 1) {
        const uint32_t i = __ffs(pick) - 1;
        const uint32_t di = __shfl_sync(kFull, d, i), ri = __shfl_sync(kFull, r, i);
        if (lane == src.n) { src.row = ri; src.start = src.total; src.info = (uint32_t)s << 5 | i; }
        src.total += di;
        ++src.n;
    }
    return true;
}

// Collects the universe of the node (S, list 0, list 1) and the rows of its
// outsiders; `top` is the first free arena word.  False (nothing changed): a
// side's outsiders are not bounded by rows (S_o has at most k members, none
// saturated), the rows are too long, or the arena has no room for outside
// vertices past the 32 per side that the lanes hold.
__device__ __forceinline__ bool bits_collect(Ctx& t, Bits& b, BitSources& src, const uint32_t* l0,
                                             uint32_t n0, const uint32_t* l1, uint32_t n1, uint32_t top) {
    const GraphView& g = t.g;
    const uint32_t lane = t.lane, k = t.k;
    BitShared& sh = *b.sh;
    const uint32_t mu = t.nss.a, mv = t.nss.b;
    b.nu = mu + n0;
    b.nv = mv + n1;
    // members to their lanes, with their miss counts (the stack's words serve
    // as scratch until the search starts)
    uint32_t* smc = reinterpret_cast<uint32_t*>(sh.stack);
    uint32_t cu = 0, cv = 0;
    #pragma unroll 1
    for (uint32_t base = 0; base < t.ns; base += 32) {
        const uint32_t i = base + lane;
        const bool in = i < t.ns;
        const uint32_t v = in ? t.sid[i] : 0u;
        const bool isv = in && side_of(g, v);
        const uint32_t bv = __ballot_sync(kFull, isv), bu = __ballot_sync(kFull, in && !isv);
        if (in) {
            const uint32_t at = isv ? 32 + cv + __popc(bv & lanemask_lt()) : cu + __popc(bu & lanemask_lt());
            sh.ids[at] = v;
            smc[at] = t.smc[i];
        }
        cu += __popc(bu);
        cv += __popc(bv);
    }
    if (lane < n0) sh.ids[mu + lane] = l0[2 * lane];
    if (lane < n1) sh.ids[32 + mv + lane] = l1[2 * lane];
    __syncwarp();
    b.iu = mu < 32 ? (1u << mu) - 1u : kFull;
    b.iv = mv < 32 ? (1u << mv) - 1u : kFull;
    b.su = __ballot_sync(kFull, lane < mu && smc[lane] >= k);
    b.sv = __ballot_sync(kFull, lane < mv && smc[32 + lane] >= k);
    uint32_t du = 0, dv = 0, ru = 0, rv = 0;
    if (lane < mu) { const uint32_t v = sh.ids[lane]; ru = g.off[v]; du = g.off[v + 1] - ru; }
    if (lane < mv) { const uint32_t v = sh.ids[32 + lane]; rv = g.off[v]; dv = g.off[v + 1] - rv; }
    // U outsiders (s = 0) come from V members' rows and the other way round
    src.start = kFull;
    src.n = src.total = 0;
    #pragma unroll 1
    for (int s = 0; s < 2; ++s)
        if (!bits_source(t, src, s, s ? b.iu : b.iv, s ? b.su : b.sv, s ? du : dv, s ? ru : rv)) return false;
    b.over = top;
    b.lanes = false;
    return src.total <= 32 || top + (unsigned long long)src.total <= t.cap;
}

// Starts the search of the collected universe (ids, sizes, I, saturated
// members, sources): miss masks, outside vertices.  False: there is nothing
// to search, C is empty and an outside vertex can join.
__device__ __forceinline__ bool bits_start(Ctx& t, Bits& b, const BitSources& src) {
    const GraphView& g = t.g;
    const uint32_t lane = t.lane, k = t.k;
    BitShared& sh = *b.sh;
    const uint32_t nu = b.nu, nv = b.nv;
    const uint32_t uid = lane < nu ? sh.ids[lane] : 0u;
    const uint32_t vid = lane < nv ? sh.ids[32 + lane] : 0u;
    b.cu = (nu < 32 ? (1u << nu) - 1u : kFull) & ~b.iu;
    b.cv = (nv < 32 ? (1u << nv) - 1u : kFull) & ~b.iv;
    const bool leaf = !(b.cu | b.cv);
    if (lane == 0) t.work += src.total;

    // miss masks: one lane group per U vertex, over the V vertices
    b.um = b.vm = 0;
    {
        const Groups gr = make_groups(nu, nv, lane);
        const uint32_t gm = gr.lg == 5 ? kFull : (1u << gr.G) - 1u;
        #pragma unroll 1
        for (uint32_t rb = 0; rb < nu; rb += gr.rows) {
            const uint32_t row = rb + gr.row;
            const uint32_t x = __shfl_sync(kFull, uid, row & 31u);
            #pragma unroll 1
            for (uint32_t cb = 0; cb < nv; cb += gr.G) {
                const uint32_t col = cb + gr.slot;
                const uint32_t y = __shfl_sync(kFull, vid, col & 31u);
                const bool miss = row < nu && col < nv && !adj_test(t, x, y);
                const uint32_t mm = __ballot_sync(kFull, miss);
                const uint32_t mine = lane - rb;      // this lane's U vertex, as a row of the pass
                if (mine < gr.rows) b.um |= ((mm >> (mine << gr.lg)) & gm) << cb;
            }
        }
        #pragma unroll 1
        for (uint32_t j = 0; j < nu; ++j)
            b.vm |= ((__shfl_sync(kFull, b.um, j) >> lane) & 1u) << j;
    }

    // outside vertices: one lane group per row entry, over the universe
    uint32_t* out = reinterpret_cast<uint32_t*>(sh.found);   // first 32 per side (scratch)
    uint32_t nou = 0, nov = 0;
    const uint32_t wide = nu > nv ? nu : nv;
    const Groups gr = make_groups(src.total, wide, lane);
    const uint32_t gm = gr.lg == 5 ? kFull : (1u << gr.G) - 1u;
    #pragma unroll 1
    for (uint32_t base = 0; base < src.total; base += gr.rows) {
        const uint32_t p = base + gr.row;
        const bool live = p < src.total;
        uint32_t start = 0, row = 0, info = 0, before = 0;
        #pragma unroll 1
        for (uint32_t i = 0; i < src.n; ++i) {
            const uint32_t st = __shfl_sync(kFull, src.start, i), rw = __shfl_sync(kFull, src.row, i);
            const uint32_t in = __shfl_sync(kFull, src.info, i);
            if (p >= st) {
                // the sources of the same side before this one
                if (i && (info >> 5) == (in >> 5)) before |= 1u << (info & 31u);
                else before = 0;
                start = st; row = rw; info = in;
            }
        }
        const bool s = info >> 5;
        const uint32_t e = live ? g.adj[row + (p - start)] : 0u;
        const uint32_t mem = s ? b.iu : b.iv, sat = s ? b.su : b.sv;
        bool in = false, dead = !live;
        uint32_t m = 0;
        #pragma unroll 1
        for (uint32_t cb = 0; cb < wide; cb += gr.G) {
            const uint32_t col = cb + gr.slot;
            const uint32_t xu = __shfl_sync(kFull, uid, col & 31u), xv = __shfl_sync(kFull, vid, col & 31u);
            in |= col < (s ? nv : nu) && (s ? xv : xu) == e;
            const bool miss = !dead && !in && col < (s ? nu : nv) && !adj_test(t, e, s ? xu : xv);
            const uint32_t mm = __ballot_sync(kFull, miss);
            m |= ((mm >> (lane & ~(gr.G - 1u))) & gm) << cb;
            dead = dead || (uint32_t)__popc(m & mem) > k || (m & sat);
        }
        in = group_any(in, gr);
        // an entry found in an earlier source's row is taken there
        const bool keep = gr.slot == 0 && !dead && !in && !(before & ~m);
        const uint32_t ku = __ballot_sync(kFull, keep && !s), kv = __ballot_sync(kFull, keep && s);
        if (leaf && (ku | kv)) return false;
        if (keep) {
            const uint32_t r = s ? nov + __popc(kv & lanemask_lt()) : nou + __popc(ku & lanemask_lt());
            if (r < 32) out[s ? 32 + r : r] = m;
            else if (s) t.arena[t.cap - 1 - (r - 32)] = m;
            else t.arena[b.over + (r - 32)] = m;
        }
        nou += __popc(ku);
        nov += __popc(kv);
    }
    __syncwarp();
    b.ou = lane < nou ? out[lane] : 0u;
    b.ov = lane < nov ? out[32 + lane] : 0u;
    b.nou = nou; b.nov = nov;
    b.hashed = false;
    b.nfound = 0;
    b.sp = b.bottom = 0;
    b.active = true;
    __syncwarp();
    return true;
}

// Count mode: hashes the buffered results, one per lane.
__device__ __forceinline__ void bits_flush(Ctx& t, Bits& b) {
    BitShared& sh = *b.sh;
    if (!b.hashed) {
        b.hashed = true;
        const uint32_t lane = t.lane;
        #pragma unroll 1
        for (uint32_t i = lane; i < 64; i += 32) {
            if ((i & 31u) < (i < 32 ? b.nu : b.nv)) {
                const unsigned long long e = elem_a(sh.ids[i]);
                sh.ea[i] = e;
                sh.eb[i] = elem_b(e);
            }
        }
    }
    __syncwarp();
    #pragma unroll 1
    for (uint32_t base = 0; base < b.nfound; base += 32) {
        unsigned long long h1 = 0, h2 = 0;
        if (base + t.lane < b.nfound) {
            const uint2 r = sh.found[base + t.lane];
            unsigned long long x = 0, y = 0;
            #pragma unroll 1
            for (uint32_t m = r.x; m; m &= m - 1) { x += sh.ea[__ffs(m) - 1]; y += sh.eb[__ffs(m) - 1]; }
            #pragma unroll 1
            for (uint32_t m = r.y; m; m &= m - 1) { x += sh.ea[31 + __ffs(m)]; y += sh.eb[31 + __ffs(m)]; }
            h1 = final_h1(x, __popc(r.x), __popc(r.y));
            h2 = final_h2(y, __popc(r.x), __popc(r.y));
        }
        t.hsum += warp_sum64(h1);
        t.hxor ^= warp_xor64(h2);
    }
    t.cnt += b.nfound;
    b.nfound = 0;
    __syncwarp();
}

// Takes the results of the lanes with `hit` (U mask lu, V mask lv).  Count
// mode buffers them.  Record mode reserves room for all of them at once (no
// room: nothing is written, false), counts them (exact limit: past it, skip
// records) and writes them, one lane per record.
template <bool kRec>
__device__ __forceinline__ bool bits_take(Ctx& t, const Outputs& o, Bits& b, bool hit, uint32_t lu,
                                          uint32_t lv) {
    BitShared& sh = *b.sh;
    const uint32_t who = __ballot_sync(kFull, hit);
    if (!who) return true;
    const uint32_t rank = __popc(who & lanemask_lt()), n = __popc(who);
    if (!kRec) {
        if (hit) sh.found[b.nfound + rank] = make_uint2(lu, lv);
        b.nfound += n;   // at most 32 + 32 (bits_run hashes them past 32)
        return true;
    }
    const uint32_t nx = __popc(lu), ny = __popc(lv);
    uint32_t at = hit ? 2 + nx + ny : 0u;
    const uint32_t mine = at;
    #pragma unroll 1
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_up_sync(kFull, at, d);
        if (t.lane >= d) at += x;
    }
    const uint32_t words = __shfl_sync(kFull, at, 31);
    at -= mine;
    unsigned long long pos = 0, c0 = 0;
    int room = 0;
    if (t.lane == 0) {
        pos = atomicAdd(o.out_pos, (unsigned long long)words);
        room = pos + words <= o.out_cap;
        if (!room) {
            atomicMax(o.out_fail, ~pos);
        } else {
            c0 = atomicAdd(o.count, (unsigned long long)n);
            if (o.limit && c0 + n >= o.limit) atomicExch(o.stop, 1);
        }
    }
    if (!bcast(room)) return false;
    pos = bcast(pos);
    c0 = bcast(c0);
    unsigned long long h1 = 0, h2 = 0;
    if (hit) {
        uint32_t* r = o.out_buf + pos + at;
        if (o.limit && c0 + rank >= o.limit) {
            r[0] = 0xFFFFFFFFu;   // past the limit: a skip record of the same length
            r[1] = nx + ny;
        } else {
            unsigned long long x = 0, y = 0;
            uint32_t w = 2;
            #pragma unroll 1
            for (uint32_t i = 0; i < 64; ++i) {
                if (!(((i < 32 ? lu : lv) >> (i & 31u)) & 1u)) continue;
                const uint32_t v = sh.ids[i];
                const unsigned long long e = elem_a(v);
                x += e;
                y += elem_b(e);
                r[w++] = v;
            }
            r[0] = nx;
            r[1] = ny;
            h1 = final_h1(x, nx, ny);
            h2 = final_h2(y, nx, ny);
        }
    }
    h1 = warp_sum64(h1);
    h2 = warp_xor64(h2);
    if (t.lane == 0) {
        atomicAdd(o.hash_sum, h1);
        atomicXor(o.hash_xor, h2);
    }
    __syncwarp();
    return true;
}

// Subsets T of C, one per lane: is I u T (masks *ru, *rv) a result?  *feasible:
// how many of them are k-biplexes -- the nodes of their set-enumeration tree,
// which this one node stands for.
__device__ __forceinline__ bool bits_subsets(Ctx& t, Bits& b, uint32_t* ru, uint32_t* rv,
                                             uint32_t* feasible) {
    const uint32_t lane = t.lane, k = t.k;
    uint32_t lu = b.iu, lv = b.iv, j = 0;
    #pragma unroll 1
    for (uint32_t y = b.cu; y; y &= y - 1, ++j) lu |= ((lane >> j) & 1u) ? (y & (0u - y)) : 0u;
    #pragma unroll 1
    for (uint32_t y = b.cv; y; y &= y - 1, ++j) lv |= ((lane >> j) & 1u) ? (y & (0u - y)) : 0u;
    bool alive = (lane >> j) == 0;
    uint32_t hu = 0, hv = 0;     // blockers: k misses already
    #pragma unroll 1
    for (uint32_t y = b.iu | b.cu; y; y &= y - 1) {
        const uint32_t i = __ffs(y) - 1;
        const uint32_t c = __popc(__shfl_sync(kFull, b.um, i) & lv);
        if ((lu >> i) & 1u) {
            alive = alive && c <= k;
            hu |= c >= k ? 1u << i : 0u;
        }
    }
    #pragma unroll 1
    for (uint32_t y = b.iv | b.cv; y; y &= y - 1) {
        const uint32_t i = __ffs(y) - 1;
        const uint32_t c = __popc(__shfl_sync(kFull, b.vm, i) & lu);
        if ((lv >> i) & 1u) {
            alive = alive && c <= k;
            hv |= c >= k ? 1u << i : 0u;
        }
    }
    *feasible = __popc(__ballot_sync(kFull, alive));
    // nothing outside may join: the universe's other vertices, the outsiders
    #pragma unroll 1
    for (uint32_t y = (b.nu < 32 ? (1u << b.nu) - 1u : kFull) & ~b.iu; y; y &= y - 1) {
        const uint32_t i = __ffs(y) - 1;
        const uint32_t m = __shfl_sync(kFull, b.um, i);
        if (!((lu >> i) & 1u) && (uint32_t)__popc(m & lv) <= k && !(m & hv)) alive = false;
    }
    #pragma unroll 1
    for (uint32_t y = (b.nv < 32 ? (1u << b.nv) - 1u : kFull) & ~b.iv; y; y &= y - 1) {
        const uint32_t i = __ffs(y) - 1;
        const uint32_t m = __shfl_sync(kFull, b.vm, i);
        if (!((lv >> i) & 1u) && (uint32_t)__popc(m & lu) <= k && !(m & hu)) alive = false;
    }
    #pragma unroll 1
    for (uint32_t r = 0; r < b.nou; ++r) {
        const uint32_t x = __shfl_sync(kFull, b.ou, r & 31u);
        const uint32_t m = r < 32 ? x : bits_over_u(t, b, r);
        if ((uint32_t)__popc(m & lv) <= k && !(m & hv)) alive = false;
    }
    #pragma unroll 1
    for (uint32_t r = 0; r < b.nov; ++r) {
        const uint32_t x = __shfl_sync(kFull, b.ov, r & 31u);
        const uint32_t m = r < 32 ? x : bits_over_v(t, b, r);
        if ((uint32_t)__popc(m & lu) <= k && !(m & hu)) alive = false;
    }
    *ru = lu;
    *rv = lv;
    return alive && lv != 0;
}

// Looks at up to kBitsBudget states; *nodes_out receives the child states
// entered.  False: a state's records found no room (record mode); that state
// is still (iu, iv, cu, cv).  The search is over when b.active is false.
template <bool kRec>
__device__ __forceinline__ bool bits_run(Ctx& t, const Outputs& o, Bits& b, uint32_t* nodes_out) {
    const uint32_t lane = t.lane, k = t.k;
    uint32_t nodes = 0;
    bool room = true;
    #pragma unroll 1
    for (uint32_t step = 0;;) {
        if (!kRec && b.nfound > (b.active ? 32u : 0u)) bits_flush(t, b);
        if (!room || !b.active || step++ == kBitsBudget) break;
        const uint32_t lu = b.iu | b.cu, lv = b.iv | b.cv;
        const uint32_t tu = __popc(b.um & lv), tv = __popc(b.vm & lu);
        const bool inu = (lu >> lane) & 1u, inv = (lv >> lane) & 1u;
        const uint32_t hu = __ballot_sync(kFull, inu && tu >= k), hv = __ballot_sync(kFull, inv && tv >= k);
        // a vertex outside S u C that can join every leaf below?
        bool add = (lane < b.nu && !inu && tu <= k && !(b.um & hv)) ||
                   (lane < b.nv && !inv && tv <= k && !(b.vm & hu)) ||
                   (lane < b.nou && (uint32_t)__popc(b.ou & lv) <= k && !(b.ou & hv)) ||
                   (lane < b.nov && (uint32_t)__popc(b.ov & lu) <= k && !(b.ov & hu));
        #pragma unroll 1
        for (uint32_t r = 32 + lane; r < b.nou; r += 32) {
            const uint32_t m = bits_over_u(t, b, r);
            add |= (uint32_t)__popc(m & lv) <= k && !(m & hv);
        }
        #pragma unroll 1
        for (uint32_t r = 32 + lane; r < b.nov; r += 32) {
            const uint32_t m = bits_over_v(t, b, r);
            add |= (uint32_t)__popc(m & lu) <= k && !(m & hu);
        }
        bool down = false;
        if (!__any_sync(kFull, add) && lv) {
            const uint32_t bu = __ballot_sync(kFull, inu && tu > k), bv = __ballot_sync(kFull, inv && tv > k);
            bool hit = lane == 0;      // S u C itself, when it is a k-biplex: nothing can join it
            uint32_t ru = lu, rv = lv, extra = 0;
            if (bu | bv) {
                // candidates in every maximal leaf below
                const uint32_t fu = __ballot_sync(kFull, ((b.cu >> lane) & 1u) && tu <= k && !(b.um & bv));
                const uint32_t fv = __ballot_sync(kFull, ((b.cv >> lane) & 1u) && tv <= k && !(b.vm & bu));
                b.iu |= fu; b.cu &= ~fu;
                b.iv |= fv; b.cv &= ~fv;
                if ((uint32_t)(__popc(b.cu) + __popc(b.cv)) <= kBitsSubset && (!kRec || o.out_cap >= 8192)) {
                    uint32_t feasible;
                    hit = bits_subsets(t, b, &ru, &rv, &feasible);
                    extra = feasible - 1;
                } else {
                    // the included vertex with the most misses, over k: at most k
                    // of them can stay, so branch on a candidate it misses (if no
                    // included one is over k, on any), the one with the most misses
                    const uint32_t wu = (((b.iu & bu) >> lane) & 1u) ? (tu << 6 | (63u - lane)) : 0u;
                    const uint32_t wv = (((b.iv & bv) >> lane) & 1u) ? (tv << 6 | (31u - lane)) : 0u;
                    const uint32_t worst = __reduce_max_sync(kFull, wu > wv ? wu : wv);
                    const uint32_t who = 63u - (worst & 63u);
                    const uint32_t xm = __shfl_sync(kFull, b.um, who & 31u), ym = __shfl_sync(kFull, b.vm, who & 31u);
                    const uint32_t pu = b.cu & (!worst ? kFull : who < 32 ? 0u : ym);
                    const uint32_t pv = b.cv & (!worst ? kFull : who < 32 ? xm : 0u);
                    const uint32_t ku = ((pu >> lane) & 1u) ? (tu << 6 | (63u - lane)) : 0u;
                    const uint32_t kv = ((pv >> lane) & 1u) ? (tv << 6 | (31u - lane)) : 0u;
                    const uint32_t at = 63u - (__reduce_max_sync(kFull, ku > kv ? ku : kv) & 63u);
                    const uint32_t bit = 1u << (at & 31u);
                    if (at < 32) b.cu &= ~bit; else b.cv &= ~bit;
                    if (lane == 0) b.sh->stack[b.sp] = make_uint4(b.iu, b.iv, b.cu, b.cv);
                    ++b.sp;
                    if (at < 32) b.iu |= bit; else b.iv |= bit;
                    // what stays compatible
                    const uint32_t xu = __popc(b.um & b.iv), xv = __popc(b.vm & b.iu);
                    const uint32_t su = __ballot_sync(kFull, ((b.iu >> lane) & 1u) && xu >= k);
                    const uint32_t sv = __ballot_sync(kFull, ((b.iv >> lane) & 1u) && xv >= k);
                    b.cu &= __ballot_sync(kFull, xu <= k && !(b.um & sv));
                    b.cv &= __ballot_sync(kFull, xv <= k && !(b.vm & su));
                    down = true;
                }
            }
            if (!down) room = bits_take<kRec>(t, o, b, hit, ru, rv);
            if (room) nodes += extra;
        }
        if (down) {
            ++nodes;
        } else if (room) {
            // the next left-out state
            if (b.sp == b.bottom) {
                b.active = false;
            } else {
                --b.sp;
                __syncwarp();
                const uint4 st = b.sh->stack[b.sp];
                __syncwarp();
                b.iu = st.x; b.iv = st.y; b.cu = st.z; b.cv = st.w;
                ++nodes;
            }
        }
    }
    *nodes_out = nodes;
    return room;
}

// ----------------------------------------------------------------- records of states

__device__ __forceinline__ uint32_t bits_words(const uint4& st) {
    return kRecHeader + F_WORDS + 2u * (__popc(st.x) + __popc(st.y) + __popc(st.z) + __popc(st.w));
}

// Writes state st as the record of a node that has not been entered.
__device__ __forceinline__ void bits_record(Ctx& t, const Bits& b, const uint4& st, uint32_t* r) {
    const uint32_t lane = t.lane;
    const uint32_t nx = __popc(st.x), ns = nx + __popc(st.y), c0 = __popc(st.z), c1 = __popc(st.w);
    uint32_t* rs = r + kRecHeader;
    uint32_t* fr = rs + 2 * ns;
    uint32_t* lr = fr + F_WORDS;
    const uint32_t uid = b.sh->ids[lane], vid = b.sh->ids[32 + lane];
    const uint32_t xu = __popc(b.um & st.y), xv = __popc(b.vm & st.x);
    if (lane == 0) { r[0] = ns; r[1] = c0; r[2] = c1; r[3] = t.gid; }
    if ((st.x >> lane) & 1u) {
        const uint32_t at = __popc(st.x & lanemask_lt());
        rs[at] = uid; rs[ns + at] = xu;
    }
    if ((st.y >> lane) & 1u) {
        const uint32_t at = nx + __popc(st.y & lanemask_lt());
        rs[at] = vid; rs[ns + at] = xv;
    }
    if (lane < F_WORDS) fr[lane] = lane == F_NS ? ns : lane == F_END ? 0xFFFFFFFFu : 0u;
    if ((st.z >> lane) & 1u) {
        const uint32_t at = __popc(st.z & lanemask_lt());
        lr[2 * at] = uid; lr[2 * at + 1] = xu;
    }
    if ((st.w >> lane) & 1u) {
        const uint32_t at = c0 + __popc(st.w & lanemask_lt());
        lr[2 * at] = vid; lr[2 * at + 1] = xv;
    }
}

// Hands the oldest left-out state to a waiting warp.  False: none is left, or
// it is too small to be worth a record, or the buffer is full.
__device__ __forceinline__ bool bits_donate(Ctx& t, const Donation& db, Bits& b) {
    if (b.bottom == b.sp) return false;
    __syncwarp();
    const uint4 st = b.sh->stack[b.bottom];
    if ((uint32_t)(__popc(st.z) + __popc(st.w)) <= kBitsSubset) return false;
    const uint32_t words = bits_words(st);
    unsigned long long w0 = 0, slot = 0;
    int ok = 0;
    if (t.lane == 0) {
        w0 = atomicAdd(db.used, (unsigned long long)words);
        if (w0 + words <= db.word_cap) {
            slot = atomicAdd(db.tail, 1ull);
            ok = slot < db.idx_cap;
        }
        if (!ok) atomicExch(db.full, 1);
    }
    if (!bcast(ok)) return false;
    w0 = bcast(w0);
    bits_record(t, b, st, db.words + w0);
    __threadfence();
    __syncwarp();
    if (t.lane == 0) {
        atomicAdd(db.outstanding, 1ull);   // before it can finish
        atomicAdd(db.donated, 1ull);
        __threadfence();
        atomicExch(db.idx + slot, db.tag | (w0 + 1));
    }
    ++b.bottom;
    __syncwarp();
    return true;
}

// Writes the current state and every left-out one as tasks of the next round;
// all or nothing.
__device__ __forceinline__ bool bits_split(Ctx& t, const SplitBuf& sb, Bits& b) {
    __syncwarp();
    if (t.lane == 0) b.sh->stack[b.sp] = make_uint4(b.iu, b.iv, b.cu, b.cv);
    __syncwarp();
    unsigned long long words = 0;
    #pragma unroll 1
    for (uint32_t i = b.bottom; i <= b.sp; ++i) words += bits_words(b.sh->stack[i]);
    unsigned long long w0 = 0, r0 = 0;
    if (!reserve_records(t, sb, words, b.sp + 1 - b.bottom, &w0, &r0)) return false;
    #pragma unroll 1
    for (uint32_t i = b.bottom; i <= b.sp; ++i) {
        const uint4 st = b.sh->stack[i];
        bits_record(t, b, st, sb.words + w0);
        if (t.lane == 0) sb.idx[r0] = w0;
        w0 += bits_words(st);
        ++r0;
    }
    __syncwarp();
    b.active = false;
    return true;
}

}  // namespace warp
}  // namespace gmk

// Children of a global side, one per lane (sm_100a device code).
//
// A frame that iterates a global side s tries every vertex c of a long id
// range, and almost every child S + c is tiny: c misses the members of S on
// the other side o, one of them reaches k misses, so both candidate sides turn
// local with a handful of entries, and often none.  Built one by one, such a
// child costs a frame, two lists and a node (1 000 warp instructions and
// more); here 32 consecutive children are decided at once, each by its lane:
//
//   * which members c misses: the members' sorted rows are walked along with
//     the range (a cursor each), so no hash probe is needed;
//   * z0, the lowest-degree member of S_o with one miss left, must be missed
//     by c; then every vertex of side s that may still join lies in z0's row.
//     That row is filtered once per call into a list (ws) of ids and masks of
//     missed members: entries above c are candidates, the others outsiders;
//   * vertices of side o come from the row of a saturated member of S_s
//     (filtered once into the list wo, with the misses between the two lists,
//     and their rows walked along as the members' are: no probe is left in the
//     block) or, when c itself has k misses, from c's own row, walked by its
//     lane;
//   * with m <= kLaneC candidates, every subset T is tested.  All lanes are at
//     the same T.  A vertex is a bit: members 0..ns-1, c at ns, candidates
//     from 16; miss counts of all vertices are kept bit-sliced in four words,
//     so adding a candidate is a ripple add of its miss mask, and the tests
//     "more than k" and "at least k" are a handful of logic operations.
//
// Children whose sides both turn local, but with more candidates or outsiders
// or a longer row, go to the bit-mask search straight from here (lane_child):
// their universe comes from the same lists and rows, so no frame is built.  The
// rest (a side stays global, c adjacent to z0, a side of more than 32 vertices)
// is built the usual way, and so are all children of a frame that has no z0, too
// long a row or list, or more than 15 members (FL_ONE0, FL_ONE1).  Both kinds are left pending in the frame, as a mask
// in the words of the list that a global side does not have.  Where a child
// goes depends on the frame and the child alone, so the tree does not depend on
// how its range was cut.
#pragma once

namespace gmk {
namespace warp {

// (k = 1, cl20k: 3 candidates 1.3x, cl50k 1.8x slower than 4, 5 no faster; rows of
// 64 no faster than 32)
constexpr uint32_t kLaneC = 4;              // candidates of a child, at most
constexpr uint32_t kLaneO = 8;              // outsiders of a child, at most
constexpr uint32_t kLaneRow = 32;           // length of a row walked by one lane
constexpr uint32_t kLaneList = 64;          // entries of a shared list
constexpr uint32_t kLaneScan = 512;         // length of the row a list is filtered from
constexpr uint32_t kLaneBlocks = 4;         // blocks of 32 children per call (1: cl500k 1.45x slower)
constexpr uint32_t kLaneBits = 1024;        // row of a child that goes to the bit search

// Shared memory of one warp's lane blocks: what holds for a frame (its next
// blocks and their pending children use it as long as no other frame's did), ...
struct LaneShared {
    uint32_t ids[16], off[16], deg[16];     // the members, their rows
    uint32_t cursor[16];                    // S_o's rows: the first entry >= the next block's base
    uint32_t ws_id[kLaneList], ws_m[kLaneList];
    uint32_t wo_id[kLaneRow], wo_m[kLaneRow];
    uint32_t wo_at[kLaneRow], wo_end[kLaneRow];   // wo's rows, as cursors into adj
    uint32_t ws_miss[kLaneList];            // wo entries that each ws entry misses
    uint32_t own, opp, sat0, ss;            // members on c's side, on the other; one miss left; at k
    uint32_t z0, zs;                        // lowest-degree members of sat0 and ss (zs 32: none)
    uint32_t nws, nwo, listed;
    uint32_t miss[4];                       // the members' miss counts, bit-sliced
    unsigned long long a, b;                // hash sums of S
    uint32_t mc[32];                        // members that each child of the last block misses
};
// ... and what only deciding a block needs (the bit search's words).
struct LaneScratch {
    uint32_t cid[kLaneC][32], cw[kLaneC][32];
    uint32_t cq[kLaneC][32];                // ws position of the candidates of c's side
    uint32_t ow[kLaneO][32];
};

// The frame that the lists are for, its next position, and the last block's
// pending children for the bit search.
struct LaneCtx {
    uint32_t cur, next, direct;
};

// Four bit-sliced counters per bit position.
struct Planes {
    uint32_t a, b, c, d;
    __device__ __forceinline__ void add(uint32_t m) {
        uint32_t x = a & m; a ^= m; m = x;
        x = b & m; b ^= m; m = x;
        x = c & m; c ^= m;
        d ^= x;
    }
    // positions with counts above / equal to k
    __device__ __forceinline__ void compare(uint32_t k, uint32_t& gt, uint32_t& eq) const {
        const uint32_t k3 = 0u - ((k >> 3) & 1u), k2 = 0u - ((k >> 2) & 1u);
        const uint32_t k1 = 0u - ((k >> 1) & 1u), k0 = 0u - (k & 1u);
        gt = d & ~k3;              eq = ~(d ^ k3);
        gt |= eq & c & ~k2;        eq &= ~(c ^ k2);
        gt |= eq & b & ~k1;        eq &= ~(b ^ k1);
        gt |= eq & a & ~k0;        eq &= ~(a ^ k0);
    }
};

// First position of the sorted row [0, d) whose entry is >= v (warp).
__device__ __forceinline__ uint32_t lower_bound_warp(const uint32_t* row, uint32_t d, uint32_t v,
                                                     uint32_t lane) {
    uint32_t lo = 0, hi = d;
    #pragma unroll 1
    while (hi - lo > 32) {
        // 32 interior probes; the answer lies in the gap after the last one below v
        const uint32_t step = (hi - lo) / 33 + 1;
        const unsigned long long p = lo + (unsigned long long)(lane + 1) * step - 1;
        const uint32_t below = __popc(__ballot_sync(kFull, p < hi && row[p] < v));
        const uint32_t nlo = lo + below * step;
        const unsigned long long nhi = lo + (unsigned long long)(below + 1) * step - 1;
        hi = below < 32 && nhi < hi ? (uint32_t)nhi : hi;
        lo = nlo < hi ? nlo : hi;
    }
    return lo + __popc(__ballot_sync(kFull, lo + lane < hi && row[lo + lane] < v));
}

// Filters the row of member z (offset, length d) into a list: vertices outside
// S with at most k misses among the members `opp` of the other side, none of
// them in `sat`.  False: more than kLaneList entries.
__device__ __forceinline__ bool lane_list(Ctx& t, uint32_t off, uint32_t d, uint32_t own, uint32_t opp,
                                          uint32_t z, uint32_t sat, uint32_t* out_id,
                                          uint32_t* out_m, const uint32_t* ids, uint32_t* n_out) {
    const uint32_t* row = t.g.adj + off;
    uint32_t n = 0;
    if (t.lane == 0) t.work += d;
    #pragma unroll 1
    for (uint32_t base = 0; base < d; base += 32) {
        const uint32_t p = base + t.lane;
        bool keep = p < d;
        const uint32_t v = keep ? row[p] : 0u;
        uint32_t m = 0;
        #pragma unroll 1
        for (uint32_t y = own; y; y &= y - 1) keep = keep && v != ids[__ffs(y) - 1];
        #pragma unroll 1
        for (uint32_t y = opp & ~(1u << z); y; y &= y - 1) {
            const uint32_t i = __ffs(y) - 1;
            if (keep && !adj_test(t, v, ids[i])) m |= 1u << i;
        }
        keep = keep && (uint32_t)__popc(m) <= t.k && !(m & sat);
        const uint32_t km = __ballot_sync(kFull, keep);
        if (n + __popc(km) > kLaneList) return false;
        if (keep) {
            const uint32_t r = n + __popc(km & lanemask_lt());
            out_id[r] = v;
            out_m[r] = m;
        }
        n += __popc(km);
    }
    __syncwarp();
    *n_out = n;
    return true;
}

// Writes one lane's records (record mode).
__device__ __forceinline__ void lane_record(uint32_t* r, const uint32_t* ids, uint32_t ns, uint32_t mv,
                                            uint32_t c, int s, uint32_t cs1, const uint32_t* cid,
                                            uint32_t m, uint32_t T, uint32_t nx, uint32_t ny) {
    r[0] = nx;
    r[1] = ny;
    uint32_t px = 2, py = 2 + nx;
    #pragma unroll 1
    for (uint32_t i = 0; i < ns; ++i) {
        if ((mv >> i) & 1u) r[py++] = ids[i]; else r[px++] = ids[i];
    }
    if (s) r[py++] = c; else r[px++] = c;
    #pragma unroll 1
    for (uint32_t j = 0; j < m; ++j) {
        if (!((T >> j) & 1u)) continue;
        if ((cs1 >> j) & 1u) r[py++] = cid[j * 32]; else r[px++] = cid[j * 32];
    }
}


// Decides children of frame `cur` (header h, entered, iterating its global
// side s): the pending ones (h.cnt of that side, when a block's were handed
// on or the lists have been overwritten), or up to kLaneBlocks blocks of 32
// from h.pos, the last one the first with a child that does not fit.  Writes the
// frame's position and pending children; *nodes receives the children decided here.
// False: no block was looked at, the side's children are built one by one from
// here on (FL_ONE0 / FL_ONE1).
template <bool kRec>
__device__ __forceinline__ bool lane_blocks(Ctx& t, const Outputs& o, uint32_t cur, const Hdr& h, int s,
                                            bool opp_done, LaneCtx& lc, uint32_t* nodes) {
    const GraphView& g = t.g;
    const uint32_t lane = t.lane, k = t.k;
    LaneShared& sh = *t.lanes;
    LaneScratch& sc = *t.lane_scratch;
    const uint32_t ns = h.ns;
    const uint32_t end = h.end < side_end(g, s) ? h.end : side_end(g, s);
    const uint32_t again = h.cnt.get(s);       // pending children to look at again
    uint32_t pos = again ? h.off.get(s) : h.pos, pbase = pos, pend = 0, direct = 0, done = 0;
    const uint32_t lo_o = h.lo.get(1 - s);
    bool fits = true;
    if (again || lc.cur != cur || lc.next != pos) {
        // the members, one per lane
        pop_to(t, ns);
        fits = ns <= kLaneMembers && k <= kLaneK;
        const bool is_m = fits && lane < ns;
        const uint32_t mid = is_m ? t.sid[lane] : 0u, msc = is_m ? t.smc[lane] : 0u;
        const bool mo = is_m && side_of(g, mid) != s;
        const uint32_t opp = __ballot_sync(kFull, mo), own = __ballot_sync(kFull, is_m && !mo);
        const uint32_t sat0 = __ballot_sync(kFull, mo && msc + 1 == k);
        const uint32_t ss = __ballot_sync(kFull, is_m && !mo && msc >= k);
        uint32_t moff = 0, mdeg = 0;
        if (is_m) { moff = g.off[mid]; mdeg = g.off[mid + 1] - moff; }
        const uint32_t dk = mdeg < (1u << 26) ? mdeg << 5 | lane : kFull;
        const uint32_t zk = __reduce_min_sync(kFull, ((sat0 >> lane) & 1u) ? dk : kFull);
        const uint32_t sk = __reduce_min_sync(kFull, ((ss >> lane) & 1u) ? dk : kFull);
        const bool has_ss = sk != kFull && opp_done;
        const bool listed = has_ss && (sk >> 5) <= kLaneRow;
        fits = fits && zk != kFull && (zk >> 5) <= kLaneScan;
        if (fits) {
            __syncwarp();
            if (is_m) { sh.ids[lane] = mid; sh.off[lane] = moff; sh.deg[lane] = mdeg; }
            __syncwarp();
            // ws, then (listed) wo
            #pragma unroll 1
            for (int l = 0; l < (listed ? 2 : 1) && fits; ++l) {
                uint32_t n = 0;
                fits = lane_list(t, sh.off[(l ? sk : zk) & 31u], (l ? sk : zk) >> 5, l ? opp : own, l ? own : opp,
                                 (l ? sk : zk) & 31u, l ? ss : 0u, l ? sh.wo_id : sh.ws_id,
                                 l ? sh.wo_m : sh.ws_m, sh.ids, &n);
                if (lane == 0) { if (l) sh.nwo = n; else sh.nws = n; }
            }
        }
        if (fits) {
            const unsigned long long e = is_m ? elem_a(mid) : 0ull;
            const unsigned long long a_s = warp_sum64(e), b_s = warp_sum64(is_m ? elem_b(e) : 0ull);
            const uint32_t p0 = __ballot_sync(kFull, msc & 1u), p1 = __ballot_sync(kFull, msc & 2u);
            const uint32_t p2 = __ballot_sync(kFull, msc & 4u), p3 = __ballot_sync(kFull, msc & 8u);
            if (lane == 0) {
                sh.own = own; sh.opp = opp; sh.sat0 = sat0; sh.ss = ss;
                sh.z0 = zk & 31u;
                sh.zs = has_ss ? sk & 31u : 32u;
                sh.listed = listed;
                sh.miss[0] = p0; sh.miss[1] = p1; sh.miss[2] = p2; sh.miss[3] = p3;
                sh.a = a_s; sh.b = b_s;
            }
            if (listed) {
                // wo's rows from pos on (lane q searches row q), and the misses
                // between ws and wo, one ws entry per lane
                const uint32_t nwo = sh.nwo, nws = sh.nws;
                if (lane < nwo) {
                    const uint32_t w = sh.wo_id[lane], end_w = g.off[w + 1];
                    uint32_t lo = g.off[w], hi = end_w;
                    while (lo < hi) {
                        const uint32_t mid_w = lo + ((hi - lo) >> 1);
                        if (g.adj[mid_w] < pos) lo = mid_w + 1; else hi = mid_w;
                    }
                    sh.wo_at[lane] = lo;
                    sh.wo_end[lane] = end_w;
                }
                #pragma unroll 1
                for (uint32_t q = lane; q < nws; q += 32) {
                    const uint32_t v = sh.ws_id[q];
                    uint32_t m = 0;
                    #pragma unroll 1
                    for (uint32_t i = 0; i < nwo; ++i) m |= adj_test(t, v, sh.wo_id[i]) ? 0u : 1u << i;
                    sh.ws_miss[q] = m;
                }
            }
            // the first entries of S_o's rows that are >= pos
            #pragma unroll 1
            for (uint32_t y = opp; y; y &= y - 1) {
                const uint32_t i = __ffs(y) - 1;
                const uint32_t p = lower_bound_warp(g.adj + sh.off[i], sh.deg[i], pos, lane);
                if (lane == 0) sh.cursor[i] = p;
            }
        }
        __syncwarp();
        if (!fits) {
            lc.cur = kNoPos;
            lc.direct = 0;
            // (pending children that another warp left are used up first)
            if (lane == 0) t.arena[cur + F_FLAGS] |= again ? FL_BUILD : s ? FL_ONE1 : FL_ONE0;
            __syncwarp();
            return false;
        }
    }
    const uint32_t own = sh.own, opp = sh.opp, sat0 = sh.sat0, ss = sh.ss, z0 = sh.z0;
    const uint32_t nws = sh.nws, nwo = sh.nwo;
    const bool has_ss = sh.zs < 32, listed = sh.listed;
    const uint32_t members = (1u << ns) - 1u, in_s = members | 1u << ns;
    unsigned long long h1 = 0, h2 = 0;
    uint32_t cnt = 0;
    #pragma unroll 1
    for (uint32_t blk = 0; blk < kLaneBlocks && (again ? blk == 0 : pos < end) && !pend; ++blk) {
        const uint32_t nc = again ? 32u : end - pos < 32 ? end - pos : 32u;
        const uint32_t todo = again ? again : nc < 32 ? (1u << nc) - 1u : kFull;
        const uint32_t c = pos + lane;
        const bool live = (todo >> lane) & 1u;
        pbase = pos;
        if (!again) pos += nc;
        uint32_t coff = 0, cdeg = 0;
        // members that c misses
        uint32_t mc = 0;
        #pragma unroll 1
        for (uint32_t y = opp; y; y &= y - 1) {
            const uint32_t i = __ffs(y) - 1;
            const uint32_t at = sh.cursor[i], p = at + lane;
            const uint32_t e = p < sh.deg[i] ? g.adj[sh.off[i] + p] - pbase : kFull;
            const uint32_t adj = __reduce_or_sync(kFull, e < 32 ? 1u << e : 0u);
            if (lane == 0) sh.cursor[i] = at + __popc(adj);
            if (!((adj >> lane) & 1u)) mc |= 1u << i;
        }
        const uint32_t mcc = __popc(mc), satc = mc & sat0;
        // both sides turn local: z0 bounds c's side; c, or a saturated member
        // of its side, the other
        const bool local = live && ((satc >> z0) & 1u) && (mcc >= k || has_ss);
        if (local && !listed) {
            coff = g.off[c];
            cdeg = g.off[c + 1] - coff;
        }
        bool simple = local && (listed || (mcc >= k && cdeg <= kLaneRow));
        // candidates of c's side
        uint32_t m = 0, no = 0;
        #pragma unroll 1
        for (uint32_t q = 0; q < nws; ++q) {
            const uint32_t v = sh.ws_id[q], mv = sh.ws_m[q];
            if (local && v > c && !(mv & satc)) {
                if (m < kLaneC) { sc.cid[m][lane] = v; sc.cw[m][lane] = mv; sc.cq[m][lane] = q; }
                ++m;
            }
        }
        // for the bit search: c's side fits a universe (the other one is
        // checked when it is collected)
        const bool to_bits = local && (uint32_t)__popc(own) + 1 + m <= kBitsSide &&
                             (mcc < k || cdeg <= kLaneBits || listed);
        simple = simple && m <= kLaneC;
        const uint32_t mcs = simple ? m : 0u;
        if (!simple) m = 0;
        // the other side: candidates and outsiders
        if (listed) {
            #pragma unroll 1
            for (uint32_t q = 0; q < nwo; ++q) {
                const uint32_t at = sh.wo_at[q], p = at + lane;
                const uint32_t e = p < sh.wo_end[q] ? g.adj[p] - pbase : kFull;
                const uint32_t adj = __reduce_or_sync(kFull, e < 32 ? 1u << e : 0u);
                if (lane == 0) sh.wo_at[q] = at + __popc(adj);
                uint32_t mw = sh.wo_m[q];
                const bool a = (adj >> lane) & 1u;
                if (!a) mw |= 1u << ns;
                if (simple && (uint32_t)__popc(mw) <= k && (a || mcc < k)) {
                    #pragma unroll 1
                    for (uint32_t j = 0; j < mcs; ++j)
                        mw |= ((sh.ws_miss[sc.cq[j][lane]] >> q) & 1u) << (16 + j);
                    if (no < kLaneO) sc.ow[no][lane] = mw;
                    ++no;
                }
            }
        } else {
            const uint32_t rows = __reduce_max_sync(kFull, simple ? cdeg : 0u);
            if (simple) t.work += cdeg;
            #pragma unroll 1
            for (uint32_t p = 0; p < rows; ++p) {
                bool act = simple && p < cdeg;
                const uint32_t w = act ? g.adj[coff + p] : 0u;
                uint32_t mw = 0;
                #pragma unroll 1
                for (uint32_t y = opp; y; y &= y - 1) act = act && w != sh.ids[__ffs(y) - 1];
                #pragma unroll 1
                for (uint32_t y = own; y; y &= y - 1) {
                    const uint32_t i = __ffs(y) - 1;
                    if (act && !adj_test(t, w, sh.ids[i])) mw |= 1u << i;
                }
                if (act && (uint32_t)__popc(mw) <= k && !(mw & ss)) {
                    if (!opp_done && w > lo_o) {
                        if (m < kLaneC) { sc.cid[m][lane] = w; sc.cw[m][lane] = mw; }
                        ++m;
                    } else {
                        #pragma unroll 1
                        for (uint32_t j = 0; j < mcs; ++j)
                            if (!adj_test(t, w, sc.cid[j][lane])) mw |= 1u << (16 + j);
                        if (no < kLaneO) sc.ow[no][lane] = mw;
                        ++no;
                    }
                }
            }
        }
        if (m > kLaneC) { simple = false; m = 0; }
        // misses between the candidates of the two sides
        if (simple) {
            #pragma unroll 1
            for (uint32_t j = mcs; j < m; ++j) {
                #pragma unroll 1
                for (uint32_t i = 0; i < mcs; ++i) {
                    if (!adj_test(t, sc.cid[j][lane], sc.cid[i][lane])) {
                        sc.cw[j][lane] |= 1u << (16 + i);
                        sc.cw[i][lane] |= 1u << (16 + j);
                    }
                }
            }
        }
        // outsiders of c's side
        #pragma unroll 1
        for (uint32_t q = 0; q < nws; ++q) {
            const uint32_t v = sh.ws_id[q];
            uint32_t mv = sh.ws_m[q];
            if (simple && v < c && !(mv & satc)) {
                #pragma unroll 1
                for (uint32_t j = mcs; j < m; ++j)
                    if (!adj_test(t, v, sc.cid[j][lane])) mv |= 1u << (16 + j);
                if (no < kLaneO) sc.ow[no][lane] = mv;
                ++no;
            }
        }
        // (a child without candidates is decided by its first outsider)
        if (no > kLaneO) {
            if (m == 0) no = 1;
            else simple = false;
        }
        pend = __ballot_sync(kFull, live && !simple);
        direct = __ballot_sync(kFull, to_bits && !simple);
        if (!simple) { m = 0; no = 0; }
        // miss counts inside S + c, bit-sliced
        Planes pl{sh.miss[0], sh.miss[1], sh.miss[2], sh.miss[3]};
        pl.add(mc);
        pl.a |= (mcc & 1u) << ns;
        pl.b |= ((mcc >> 1) & 1u) << ns;
        pl.c |= ((mcc >> 2) & 1u) << ns;
        pl.d |= ((mcc >> 3) & 1u) << ns;
        #pragma unroll 1
        for (uint32_t j = 0; j < m; ++j) {
            const uint32_t x = __popc(sc.cw[j][lane] & 0xFFFFu);
            pl.a |= (x & 1u) << (16 + j);
            pl.b |= ((x >> 1) & 1u) << (16 + j);
            pl.c |= ((x >> 2) & 1u) << (16 + j);
            pl.d |= ((x >> 3) & 1u) << (16 + j);
        }
        const uint32_t mm = __reduce_max_sync(kFull, m), mno = __reduce_max_sync(kFull, no);
        const uint32_t fs = (1u << mcs) - 1u;     // candidates of c's side
        const uint32_t n_own = __popc(own) + 1, n_opp = __popc(opp);
        uint32_t found = 0;
        unsigned long long ea_c = 0, eb_c = 0;
        if (!kRec) { ea_c = elem_a(c); eb_c = elem_b(ea_c); }
        #pragma unroll 1
        for (uint32_t T = 0; T < (1u << mm); ++T) {
            bool ok = simple && (T >> m) == 0;
            Planes q = pl;
            #pragma unroll 1
            for (uint32_t y = T; y; y &= y - 1) q.add(ok ? sc.cw[__ffs(y) - 1][lane] : 0u);
            const uint32_t in_l = in_s | T << 16;
            uint32_t gt, eq;
            q.compare(k, gt, eq);
            ok = ok && !(gt & in_l);
            const uint32_t hard = (gt | eq) & in_l;
            #pragma unroll 1
            for (uint32_t j = 0; j < mm; ++j) {
                if ((T >> j) & 1u) continue;
                if (ok && j < m) {
                    const uint32_t w = sc.cw[j][lane];
                    ok = (uint32_t)__popc(w & in_l) > k || (w & hard);
                }
            }
            #pragma unroll 1
            for (uint32_t r = 0; r < mno; ++r) {
                if (ok && r < no) {
                    const uint32_t w = sc.ow[r][lane];
                    ok = (uint32_t)__popc(w & in_l) > k || (w & hard);
                }
            }
            if (ok) found |= 1u << T;
            const uint32_t who = __ballot_sync(kFull, ok);
            if (kRec || !who) continue;
            unsigned long long x = sh.a + ea_c, y = sh.b + eb_c;
            #pragma unroll 1
            for (uint32_t z = T; z; z &= z - 1) {
                const unsigned long long e = elem_a(ok ? sc.cid[__ffs(z) - 1][lane] : 0u);
                x += e;
                y += elem_b(e);
            }
            if (ok) {
                const uint32_t a = n_own + __popc(T & fs), b = n_opp + __popc(T & ~fs);
                const uint32_t nx = s ? b : a, ny = s ? a : b;
                cnt += 1;
                h1 += final_h1(x, nx, ny);
                h2 ^= final_h2(y, nx, ny);
            }
        }
        uint32_t decided = __popc(__ballot_sync(kFull, simple));
        if (kRec && __any_sync(kFull, found != 0)) {
            // room for the block's records first, then the count
            uint32_t rank = __popc(found), words = 0;
            #pragma unroll 1
            for (uint32_t x = found; x; x &= x - 1) words += 3 + ns + __popc(__ffs(x) - 1);
            const uint32_t my_n = rank, my_w = words;
            #pragma unroll 1
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t x = __shfl_up_sync(kFull, rank, d), y = __shfl_up_sync(kFull, words, d);
                if (lane >= d) { rank += x; words += y; }
            }
            const uint32_t n_all = __shfl_sync(kFull, rank, 31), w_all = __shfl_sync(kFull, words, 31);
            rank -= my_n;
            words -= my_w;
            unsigned long long at = 0, c0 = 0;
            int room = 0;
            if (lane == 0 && 2ull * w_all <= o.out_cap) {
                at = atomicAdd(o.out_pos, (unsigned long long)w_all);
                room = at + w_all <= o.out_cap;
                if (!room) {
                    atomicMax(o.out_fail, ~at);
                } else {
                    c0 = atomicAdd(o.count, (unsigned long long)n_all);
                    if (o.limit && c0 + n_all >= o.limit) atomicExch(o.stop, 1);
                }
            }
            if (!bcast(room)) {
                // nothing was written: the block's children are built the usual
                // way, whose results can be deferred one by one
                pend = todo;
                direct = 0;
                decided = 0;
            } else {
                at = bcast(at);
                c0 = bcast(c0);
                const uint32_t mv = s ? own : opp;                     // V members
                const uint32_t cs1 = s ? fs : ~fs;                     // V candidates
                uint32_t* r = o.out_buf + at + words;
                #pragma unroll 1
                for (uint32_t x = found; x; x &= x - 1) {
                    const uint32_t T = __ffs(x) - 1;
                    const uint32_t ny = __popc(mv) + (s ? 1u : 0u) + __popc(T & cs1);
                    const uint32_t nx = ns + 1 + __popc(T) - ny;
                    if (o.limit && c0 + rank++ >= o.limit) {
                        r[0] = 0xFFFFFFFFu;   // past the limit: a skip record of the same length
                        r[1] = nx + ny;
                    } else {
                        lane_record(r, sh.ids, ns, mv, c, s, cs1, &sc.cid[0][lane], m, T, nx, ny);
                        unsigned long long e = elem_a(c), u = sh.a + e, v = sh.b + elem_b(e);
                        #pragma unroll 1
                        for (uint32_t z = T; z; z &= z - 1) {
                            e = elem_a(sc.cid[__ffs(z) - 1][lane]);
                            u += e;
                            v += elem_b(e);
                        }
                        h1 += final_h1(u, nx, ny);
                        h2 ^= final_h2(v, nx, ny);
                    }
                    r += 2 + nx + ny;
                }
            }
        }
        done += decided;
        if (pend) sh.mc[lane] = mc;
        __syncwarp();
    }
    t.cnt += __reduce_add_sync(kFull, cnt);
    h1 = warp_sum64(h1);
    h2 = warp_xor64(h2);
    if (kRec) {
        if (lane == 0 && (h1 | h2)) {
            atomicAdd(o.hash_sum, h1);
            atomicXor(o.hash_xor, h2);
        }
    } else {
        t.hsum += h1;
        t.hxor ^= h2;
    }
    if (lane == 0) {
        uint32_t* f = t.arena + cur;
        if (!again) f[F_POS] = pos;
        f[F_OFF0 + s] = pbase;
        f[F_CNT0 + s] = pend;
        // none of the pending children is for the bit search: they are built
        f[F_FLAGS] = pend && !direct ? f[F_FLAGS] | FL_BUILD : f[F_FLAGS] & ~FL_BUILD;
    }
    __syncwarp();
    lc.cur = cur;
    lc.next = again ? kNoPos : pos;
    lc.direct = direct;
    *nodes = done;
    return true;
}

// Collects the universe of the pending child `bit` of the last block's frame (h:
// its header).  False: it does not
// fit, build it.
__device__ __forceinline__ bool lane_child(Ctx& t, Bits& b, BitSources& src, const Hdr& h,
                                           int s, bool opp_done, uint32_t bit) {
    const GraphView& g = t.g;
    const uint32_t lane = t.lane, k = t.k, ns = h.ns;
    const LaneShared& sh = *t.lanes;
    BitShared& bs = *b.sh;
    const uint32_t m_own = sh.own, m_opp = sh.opp, m_ss = sh.ss, nws = sh.nws, zs = sh.zs, z0 = sh.z0;
    const uint32_t c = h.off.get(s) + bit, lo_o = h.lo.get(1 - s);
    const uint32_t mc = sh.mc[bit], satc = mc & sh.sat0, mcc = __popc(mc);
    const uint32_t n_own = __popc(m_own), n_opp = __popc(m_opp);
    uint32_t* own_id = bs.ids + (s ? 32 : 0);      // c's side of the universe
    uint32_t* opp_id = bs.ids + (s ? 0 : 32);
    // members in S order, then c
    if (lane < ns) {
        if ((m_own >> lane) & 1u) own_id[__popc(m_own & lanemask_lt())] = sh.ids[lane];
        else opp_id[__popc(m_opp & lanemask_lt())] = sh.ids[lane];
    }
    if (lane == 0) own_id[n_own] = c;
    uint32_t x = n_own + 1, y = n_opp;
    // candidates of c's side: ws entries above c that miss no member at k
    #pragma unroll 1
    for (uint32_t base = 0; base < nws; base += 32) {
        const uint32_t q = base + lane;
        const bool keep = q < nws && sh.ws_id[q] > c && !(sh.ws_m[q] & satc);
        const uint32_t km = __ballot_sync(kFull, keep);
        if (x + __popc(km) > kBitsSide) return false;
        if (keep) own_id[x + __popc(km & lanemask_lt())] = sh.ws_id[q];
        x += __popc(km);
    }
    // of the other side (a first phase only): c has k misses, so they are in its row
    const uint32_t coff = g.off[c], cdeg = g.off[c + 1] - coff;
    if (!opp_done) {
        if (lane == 0) t.work += cdeg;
        #pragma unroll 1
        for (uint32_t base = 0; base < cdeg; base += 32) {
            const uint32_t p = base + lane;
            bool keep = p < cdeg;
            const uint32_t w = keep ? g.adj[coff + p] : 0u;
            keep = keep && w > lo_o;               // (S_o is not past lo_o)
            uint32_t mw = 0;
            #pragma unroll 1
            for (uint32_t z = m_own; z; z &= z - 1) {
                const uint32_t i = __ffs(z) - 1;
                if (keep && !adj_test(t, w, sh.ids[i])) mw |= 1u << i;
            }
            keep = keep && (uint32_t)__popc(mw) <= k && !(mw & m_ss);
            const uint32_t km = __ballot_sync(kFull, keep);
            if (y + __popc(km) > kBitsSide) return false;
            if (keep) opp_id[y + __popc(km & lanemask_lt())] = w;
            y += __popc(km);
        }
    }
    __syncwarp();
    // outsiders: of c's side from z0's row, of the other from c's or from the
    // saturated member's
    const uint32_t z = sh.ids[z0];
    const uint32_t zoff = g.off[z], zdeg = g.off[z + 1] - zoff;
    uint32_t ooff = coff, odeg = mcc >= k ? cdeg : kFull, oidx = n_own;
    if (zs < 32) {
        const uint32_t v = sh.ids[zs], vo = g.off[v], vd = g.off[v + 1] - vo;
        if (vd < odeg) { ooff = vo; odeg = vd; oidx = __popc(m_own & ((1u << zs) - 1u)); }
    }
    if (odeg > kBitsScanMax) return false;
    src.n = 2;
    src.total = zdeg + odeg;
    // (the outsiders of side s lie in the row of a member of the other side)
    const uint32_t zidx = __popc(m_opp & ((1u << z0) - 1u));
    src.row = lane == 0 ? zoff : ooff;
    src.start = lane == 0 ? 0u : lane == 1 ? zdeg : kFull;
    src.info = lane == 0 ? (uint32_t)s << 5 | zidx : (uint32_t)(1 - s) << 5 | oidx;
    // members with k misses in S + c
    uint32_t sat_own = 0, sat_opp = 0;
    #pragma unroll 1
    for (uint32_t m = m_ss; m; m &= m - 1) sat_own |= 1u << __popc(m_own & ((m & (0u - m)) - 1u));
    if (mcc >= k) sat_own |= 1u << n_own;
    #pragma unroll 1
    for (uint32_t m = satc; m; m &= m - 1) sat_opp |= 1u << __popc(m_opp & ((m & (0u - m)) - 1u));
    const uint32_t in_own = (2u << n_own) - 1u, in_opp = (1u << n_opp) - 1u;
    b.iu = s ? in_opp : in_own;
    b.iv = s ? in_own : in_opp;
    b.su = s ? sat_opp : sat_own;
    b.sv = s ? sat_own : sat_opp;
    b.nu = s ? y : x;
    b.nv = s ? x : y;
    b.over = h.top;
    b.lanes = true;
    return src.total <= 32 || h.top + (unsigned long long)src.total <= t.cap;
}

}  // namespace warp
}  // namespace gmk

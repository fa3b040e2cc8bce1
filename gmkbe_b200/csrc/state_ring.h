// Slots of the small graphs' shared states: a ring that tickets 0, 1, ... of a
// launch go round (host and device code, free of CUDA calls so that it is tested
// alone).
//
// Ticket t uses slot t mod slots, as its g-th user (g = t / slots).  The slot's
// mark says ready(t) once the record of ticket t is written, and ready(t) + 1
// once it is read; a donor writes over a slot when the user before has read it.
// Marks grow from launch to launch, so what earlier launches left is neither.
//
// A donor waits for the reader of ticket t - slots only, and that one runs.  A
// warp hands states on, at most kRingShare at a time, when it saw tickets waiting:
// tail < claim, at a moment after its last donation unless the ring is in its
// first round and has kRingShare free slots a warp left (it then looks at the two
// counters one after the other, which is a memory latency cheaper).  So the
// reserved tickets end in the first round, or are never more than kRingShare a
// warp ahead of the claimed ones: ticket t - slots was claimed.
//
// Why a ring: with 128 slots a warp, each used once, the rest of a longer search was
// not shared (80 x 80, density 0.35, k = 1: 146 ms, here 67; 90 x 90, 0.4: 975, 644),
// and idle warps took a subtree of over 10 s for a standstill.
// Why kRingWarp slots a warp: a reused slot costs a donation three memory
// latencies, and most runs end in the first round (58 x 58, k = 2: 183 k states
// handed on by 3 552 warps, 2.50 ms; with 16 slots a warp 2.70).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define GMK_RING_HD __host__ __device__ __forceinline__
#else
#define GMK_RING_HD inline
#endif

namespace gmk {

constexpr uint32_t kRingShare = 8;      // states handed on at a time, at most
constexpr uint32_t kRingWarp = 64;     // slots a warp, at least

struct StateRing {
    uint32_t base, shift;               // first mark of the launch; log2(slots)
    GMK_RING_HD uint32_t slots() const { return 1u << shift; }
    GMK_RING_HD uint32_t slot(unsigned long long t) const { return (uint32_t)t & (slots() - 1); }
    GMK_RING_HD uint32_t ready(unsigned long long t) const { return base + 2 * (uint32_t)(t >> shift); }
    // the first round, with more than kRingShare slots a warp left?
    GMK_RING_HD bool early(unsigned long long tail) const { return tail < slots() - slots() / 8; }
    // the first user of its slot in this launch?
    GMK_RING_HD bool first(unsigned long long t) const { return (t >> shift) == 0; }
    // has the user before ticket t (not the first) read the slot with this mark?
    GMK_RING_HD bool free(unsigned long long t, uint32_t mark) const { return mark == ready(t) - 1; }
};

// The ring of a launch of `workers` warps.  base: what ring_next gave for the
// launch before, 0 for a buffer that is new (*clear: to be zeroed first).
inline StateRing ring_begin(uint64_t workers, uint32_t base, bool* clear) {
    StateRing r{base ? base : 1u, 0};
    static_assert(kRingWarp / 8 >= kRingShare, "early() leaves kRingShare slots a warp");
    while ((1ull << r.shift) < kRingWarp * workers) ++r.shift;
    *clear = base == 0;
    return r;
}

// First mark of the launch after one that reserved `tail` tickets; 0: the marks
// are used up, clear the buffer.
inline uint32_t ring_next(const StateRing& r, unsigned long long tail) {
    const unsigned long long next = r.base + 2 * ((tail + r.slots() - 1) >> r.shift);
    return next < 1u << 31 ? (uint32_t)next : 0u;
}

}  // namespace gmk

// Growth of the cached device workspaces, and the numbers by which a launch
// recognises its own records in memory that earlier launches wrote.  Host only,
// and free of CUDA calls (they come in as functions), so that it is tested alone.
#pragma once
#include <cstddef>
#include <cstdint>

namespace gmk {

// Makes *p hold at least `need` bytes; 0 or the allocator's status.  *fresh (when
// given) is set when the memory is new: its contents are then unknown, also where
// the allocator hands the old address out again, as cudaMalloc may after a
// cudaFree.
template <class Alloc, class Release>
int grow_buffer(void** p, size_t* have, size_t need, bool* fresh, Alloc alloc, Release release) {
    if (*have >= need && *p) return 0;
    if (*p) release(*p);
    *p = nullptr;
    *have = 0;
    if (fresh) *fresh = true;
    if (const int rc = alloc(p, need)) {
        *p = nullptr;
        return rc;
    }
    *have = need;
    return 0;
}

// Number of the next launch over a buffer of records that count when they carry
// it.  last: the previous launch's (0: none, or the buffer is new); numbers run
// up to max.  *clear: the buffer is to be zeroed before the launch.
inline uint32_t next_launch(uint32_t last, uint32_t max, bool* clear) {
    *clear = last == 0 || last >= max;
    return *clear ? 1u : last + 1;
}

}  // namespace gmk

// Index arithmetic on CSR entries, shared by the kernels and checked on the host.
//
// Entries are numbered in 32 bits up to 2^32 - 1, so a list may end within a few
// entries of 2^32, and neither a position past its end nor a rounded-up length
// may be formed: they would wrap below it. Everything here is formed from
// lengths that are left.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define GCU_HD __host__ __device__ __forceinline__
#else
#define GCU_HD inline
#endif

namespace gcu {

GCU_HD uint32_t min_u32(uint32_t a, uint32_t b) { return a < b ? a : b; }

// Ranges of `size` entries that a list of d entries makes, and the c-th of them.
GCU_HD uint32_t range_count(uint32_t d, uint32_t size) { return d / size + (d % size ? 1u : 0u); }
GCU_HD uint32_t range_begin(uint32_t s, uint32_t size, uint32_t c) { return s + c * size; }
GCU_HD uint32_t range_end(uint32_t s, uint32_t d, uint32_t size, uint32_t c) {
    return s + c * size + min_u32(size, d - c * size);
}

// [x, y) cut down to its part-th piece (empty past the last).
GCU_HD void take_piece(uint32_t& x, uint32_t& y, uint32_t part, uint32_t piece) {
    const uint32_t len = y - x, lo = min_u32(len, part * piece);
    y = x + lo + min_u32(piece, len - lo);
    x += lo;
}

// Entry o + i of [s, e), or e where the list ends before (o <= e - s).
GCU_HD uint32_t entry_or_end(uint32_t s, uint32_t e, uint32_t o, uint32_t i) { return s + o + min_u32(i, e - s - o); }

// f(o) for the offsets o = 0, step, 2 step, ... below e - s.
template <class F>
GCU_HD void walk_entries(uint32_t s, uint32_t e, uint32_t step, F f) {
    const uint32_t n = e - s;
    for (uint32_t o = 0; o < n;) {
        f(o);
        if (n - o <= step) break;
        o += step;
    }
}

}  // namespace gcu

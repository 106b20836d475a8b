// Device helpers shared by the kernel files (sm_100a, 32-lane warps).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "entry_index.h"

namespace gcu {

constexpr int kWarp = 32;
constexpr unsigned kFullMask = 0xFFFFFFFFu;

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
    return v;
}

template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T w = __shfl_xor_sync(kFullMask, v, o);
        v = w < v ? w : v;
    }
    return v;
}

// Inclusive warp scan.
template <typename T>
__device__ __forceinline__ T warp_inclusive_scan(T v) {
    const unsigned lane = lane_id();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T w = __shfl_up_sync(kFullMask, v, o);
        if (lane >= static_cast<unsigned>(o)) v += w;
    }
    return v;
}

// Block-wide sum; every thread gets the result. `scratch` holds >= 32 values.
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* scratch) {
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const unsigned nwarps = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    T r = (threadIdx.x < nwarps) ? scratch[threadIdx.x] : T(0);
    if (warp == 0) r = warp_sum(r);
    if (threadIdx.x == 0) scratch[0] = r;
    __syncthreads();
    r = scratch[0];
    __syncthreads();
    return r;
}

// Streaming load that does not allocate in L1 (data read once).
__device__ __forceinline__ uint32_t ld_stream(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ uint2 ld_stream2(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ uint4 ld_stream4(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// Predicated accesses (one instruction, no branch): several of them in a row
// stay in flight together, where `if (p) x = atomicOr(...)` waits for each
// result inside its own branch (1,790 cycles for four atomics in a row in
// the BFS push, about 600 this way). Without `p` nothing is accessed and the
// result is `other`.
__device__ __forceinline__ uint32_t atomic_or_if(bool p, uint32_t* a, uint32_t bits, uint32_t other) {
    uint32_t v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\tmov.u32 %0, %4;\n\t"
                 "@q atom.global.or.b32 %0, [%2], %3;\n\t}"
                 : "=&r"(v)
                 : "r"(static_cast<uint32_t>(p)), "l"(a), "r"(bits), "r"(other)
                 : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_if(bool p, const uint32_t* a, uint32_t other) {
    uint32_t v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\tmov.u32 %0, %3;\n\t@q ld.global.u32 %0, [%2];\n\t}"
                 : "=&r"(v)
                 : "r"(static_cast<uint32_t>(p)), "l"(a), "r"(other));
    return v;
}
__device__ __forceinline__ uint32_t ld_cg_if(bool p, const uint32_t* a, uint32_t other) {
    uint32_t v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\tmov.u32 %0, %3;\n\t@q ld.global.cg.u32 %0, [%2];\n\t}"
                 : "=&r"(v)
                 : "r"(static_cast<uint32_t>(p)), "l"(a), "r"(other));
    return v;
}
__device__ __forceinline__ uint32_t ld_nc_if(bool p, const uint32_t* a, uint32_t other) {
    uint32_t v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\tmov.u32 %0, %3;\n\t@q ld.global.nc.u32 %0, [%2];\n\t}"
        : "=&r"(v)
        : "r"(static_cast<uint32_t>(p)), "l"(a), "r"(other));
    return v;
}

// One 32-byte sector (sm_100's 256-bit load; p 32-byte aligned).
__device__ __forceinline__ void ld_stream8(const uint32_t* p, uint32_t (&v)[8]) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
}

// First index in [lo, hi) with a[idx] >= val.
__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* a, uint32_t lo, uint32_t hi, uint32_t val) {
    while (lo < hi) {
        uint32_t mid = lo + ((hi - lo) >> 1);
        if (a[mid] < val)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Largest row r in [0, n) with offsets[r] <= pos (offsets non-decreasing,
// offsets[0] == 0 <= pos).
__device__ __forceinline__ uint32_t row_of_entry(const uint32_t* offsets, uint32_t n, uint32_t pos) {
    uint32_t lo = 0, hi = n;  // answer in [lo, hi)
    while (hi - lo > 1) {
        uint32_t mid = lo + ((hi - lo) >> 1);
        if (offsets[mid] <= pos)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------------- grid barrier
// Barrier over the blocks of one cooperative launch (all resident at once).
// `arrived` counts arrivals and only grows (zeroed before the launch), so a
// phase needs one atomic per block and no reset; the comparison is by signed
// difference, so the count may wrap. A block that waits for kGridSpinLimit
// polls (seconds, against phases of at most milliseconds) gives up: it raises
// `failed`, every block returns false from its barrier, and the kernel ends
// with the flag set instead of hanging. Plain loads after the barrier see
// what any block stored before it; data that changes inside the kernel must
// not be read through the read-only (nc) path.
struct GridBarrier {
    unsigned arrived;
    unsigned failed;
};
constexpr unsigned kGridSpinLimit = 1u << 25;

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add(unsigned* p, unsigned x) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}

// Every thread of the `blocks` blocks that share `bar` calls it; `phase` is the
// block's count of barriers on `bar` so far; thread 0 of every block runs after() once all have arrived
// (to fetch what the block needs into shared memory under the same block
// barrier). False: another block is missing, the kernel must return.
template <class After>
__device__ __forceinline__ bool grid_barrier(GridBarrier* bar, unsigned blocks, unsigned& phase, After after) {
    __shared__ unsigned s_ok;
    ++phase;
    if (blocks == 1) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();  // drops L1 lines that atomics have outdated
            after();
        }
        __syncthreads();
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = phase * blocks;
        red_release_add(&bar->arrived, 1u);  // after every store of the block (the block barrier above)
        unsigned ok = 1;
        for (unsigned i = 0; static_cast<int>(ld_relaxed(&bar->arrived) - target) < 0; ++i) {
            if (i >= kGridSpinLimit || ((i & 1023u) == 1023u && ld_relaxed(&bar->failed))) {
                atomicExch(&bar->failed, 1u);
                ok = 0;
                break;
            }
        }
        ld_acquire(&bar->arrived);
        after();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ bool grid_barrier(GridBarrier* bar, unsigned& phase) {
    return grid_barrier(bar, gridDim.x, phase, [] {});
}

// ---------------------------------------------------------------- entry tiles
// A block that works on a tile of consecutive CSR entries [e0, e1) finds the
// row of each entry from the row starts of the tile, staged in shared memory
// (s_start, kTile words; s_meta, 2 words); when the tile spans more rows than
// fit (runs of empty rows), each entry searches the global offsets instead.

// Largest row r in [0, n) with offsets[r] <= pos (defined above) picks, among
// empty rows that share a start, the non-empty row that holds the entry.
template <int kTile>
__device__ __forceinline__ bool stage_tile_rows(const uint32_t* __restrict__ offsets, uint32_t V, uint64_t e0,
                                                uint64_t e1, uint32_t* s_start, uint32_t* s_meta) {
    if (threadIdx.x < 2)
        s_meta[threadIdx.x] = row_of_entry(offsets, V, static_cast<uint32_t>(threadIdx.x == 0 ? e0 : e1 - 1));
    __syncthreads();
    const uint32_t r0 = s_meta[0], nrows = s_meta[1] - r0 + 1;
    const bool staged = nrows <= static_cast<uint32_t>(kTile);
    if (staged)
        for (uint32_t k = threadIdx.x; k < nrows; k += blockDim.x) s_start[k] = offsets[r0 + k];
    __syncthreads();
    return staged;
}

__device__ __forceinline__ uint32_t tile_row(const uint32_t* __restrict__ offsets, uint32_t V, const uint32_t* s_start,
                                             bool staged, uint32_t r0, uint32_t nrows, uint32_t j) {
    if (!staged) return row_of_entry(offsets, V, j);
    uint32_t lo = 0, hi = nrows;  // largest k with s_start[k] <= j
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (s_start[mid] <= j)
            lo = mid;
        else
            hi = mid;
    }
    return r0 + lo;
}

__host__ __device__ __forceinline__ uint64_t min_u64(uint64_t a, uint64_t b) { return a < b ? a : b; }

__host__ __device__ __forceinline__ uint64_t ceil_div_u64(uint64_t a, uint64_t b) { return (a + b - 1) / b; }

// Calls f(j, row) for every entry j of a CSR with V rows and E entries: each
// block takes tiles of kThreads * kItems consecutive entries (grid-stride),
// so long rows are shared by many blocks and every access to the entries is
// coalesced. All threads of the block must call it.
template <int kThreads, int kItems, class F>
__device__ __forceinline__ void for_each_entry(const uint32_t* __restrict__ offsets, uint32_t V, uint64_t E, F f) {
    constexpr int kTile = kThreads * kItems;
    __shared__ uint32_t s_start[kTile];
    __shared__ uint32_t s_meta[2];
    for (uint64_t e0 = static_cast<uint64_t>(blockIdx.x) * kTile; e0 < E;
         e0 += static_cast<uint64_t>(gridDim.x) * kTile) {
        const uint64_t e1 = min_u64(e0 + kTile, E);
        const bool staged = stage_tile_rows<kTile>(offsets, V, e0, e1, s_start, s_meta);
        const uint32_t r0 = s_meta[0], nrows = s_meta[1] - r0 + 1;
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
            const uint64_t j = e0 + q * kThreads + threadIdx.x;
            if (j < e1) f(static_cast<uint32_t>(j), tile_row(offsets, V, s_start, staged, r0, nrows,
                                                              static_cast<uint32_t>(j)));
        }
        __syncthreads();  // the staged starts are rewritten for the next tile
    }
}

}  // namespace gcu

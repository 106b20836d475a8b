// Triangle counting (symmetric CSRs, fixed schedule) and edge supports (k-truss)
// over word lists.
//
// Vertices are ranked by degree class (degree_class_order: hubs first), and
// N+(u) is the set of u's neighbours that rank below it. Hubs take most of the
// entries, so the ranks in an N+(u) crowd together: as bits of 32-rank words, a
// list of R-MAT 22 has 0.79 words per entry, and weighted by the counting work
// 2.5 times fewer words than entries (R-MAT 16: 4.3). A word costs what an entry
// cost (a load, a table lookup), so the lists are kept as (word, mask) pairs and
// an intersection is a sum of popcounts.
//
// The count is the sum over edges {u, v} of |N+(u) ∩ N+(v)|: every triangle
// once, at the edge of its two highest-ranked vertices. Each edge is counted
// from the end whose list has more words (ties: the larger id, or, with one word
// each, the higher rank), the owner: the owner's words go into a table in shared memory and the other end's words are
// streamed against it, 4, 16 or 32 lanes per list. An owner reads its neighbours
// from its own CSR row, so there are no in-lists and no oriented CSR to build.
//  * owners of up to kWarpWords words and kWarpOwnerRow neighbours: a warp each,
//    with a hash table of (word, mask);
//  * the others: CTA items of kSlice neighbours; the table is a bitmap of the
//    ranks below kBitmapRanks where the owner's rank allows, a hash table of up
//    to kHashWords words elsewhere, and for longer lists the bitmap again, one
//    window of kBitmapRanks ranks after the other.
// Only the owner's words are ever set and cleared, not the whole bitmap.
//
// Measured on one B200 against the oriented-CSR form (triangle.cu): R-MAT 16
// 3.13 -> 0.19 ms, R-MAT 22 30.7 -> 11.7 ms (count 9.6, lists 1.9), the triangles
// of 256 batched graphs 9.5 -> 3.6 ms. On the way, R-MAT 22 count: one word per
// lane and four lists in flight, 256-thread blocks 14.9 ms (76 instructions per
// 32 words, 24 % of the stalls at the items' block barriers); two words per lane
// 11.5; 128-thread blocks with a 16 KB bitmap 10.7; two lists in flight, 40
// registers 10.1; lists by length, 4 / 16 / 32 lanes each, 9.9 (with four in
// flight 13.3: a fifth fewer resident blocks). What bounds it is instruction
// issue.
//
// The support of an edge {u, v} is |N(u) ∩ N(v)|: the same sum of popcounts, kept
// per edge, over lists of all neighbours. R-MAT 18 has 622 M words to stream that
// way, 6.8 times those of the N+ lists, but each edge's sum is stored once, where
// enumerating the triangles of the oriented CSR takes three scattered atomics per
// triangle: 0.94 ms (and 0.25 ms for the lists) against 5.6 (and 0.35 for the
// CSR). A full list reaches all ranks, so the bitmap covers all vertices while it
// fits an SM's shared memory, 1.7 M of them, with the blocks as wide as it is
// large: 128 threads with 16 KB, 1024 with 208 KB.
#include <algorithm>

#include "device_common.cuh"
#include "gcu_internal.h"

namespace gcu {

namespace {

constexpr int kTwThreads = 256;
constexpr int kTwWarps = kTwThreads / 32;
constexpr int kCountThreads = 128;       // of the count
constexpr int kCountWarps = kCountThreads / 32;
constexpr int kCountCtasPerSm = 12;
constexpr uint32_t kNoWord = 0xFFFFFFFFu;
constexpr uint32_t kWarpRow = 128;       // neighbours of a row that one warp turns into words
// Words of an owner with a warp table: 64 on a large graph; 32 below
// kSmallGraph vertices, where the last owners of a few warps would be the end
// of the launch (R-MAT 16: 81 against 123 us; R-MAT 22: 10.2 against 9.9 ms).
constexpr uint32_t kWarpWords = 64, kWarpWordsSmall = 32;
constexpr uint32_t kSmallGraph = 1u << 19;
constexpr uint32_t kWarpOwnerRow = 128;  // neighbours of such an owner
constexpr uint32_t kWarpBits = 8;
constexpr int kInFlight = 2;             // lists in flight per group of lanes in the count
constexpr uint32_t kSlice = 2048;        // neighbours per CTA item
constexpr uint32_t kBitmapWords = 4096;
constexpr uint32_t kBitmapRanks = kBitmapWords * 32;
constexpr uint32_t kHashBits = 11;       // 2048 (word, mask) slots: as many bytes as the bitmap
constexpr uint32_t kHashWords = 1u << (kHashBits - 1);
constexpr size_t kSmemPerSm = size_t(227) << 10;
// Of the support's blocks (bitmap, lists in hand and 1 KB reserved each): 12 of
// 128 threads, 6 of 256, 3 of 512 or one of 1024 in an SM, by the bitmap's bytes.
constexpr size_t kBitmap128 = size_t(16) << 10, kBitmap256 = size_t(33) << 10, kBitmap512 = size_t(66) << 10;
constexpr uint32_t kMaxBitmapWords = 52u << 10;  // 1.7 M ranks
constexpr uint32_t kMaxTableWords = (1024 / 32) * (2u << kWarpBits);
static_assert((1u << kHashBits) * 2 == kBitmapWords, "one shared array for both tables");
static_assert(kCountWarps * (2u << kWarpBits) <= kBitmapWords, "the warps' tables fit the shared array");

__device__ __forceinline__ uint32_t word_slot(uint32_t word, uint32_t bits) { return (word * 2654435761u) >> (32 - bits); }

// ORs mask into the table entry of `word` (2^bits slots, never full).
__device__ __forceinline__ void table_or(uint2* table, uint32_t bits, uint32_t word, uint32_t mask) {
    const uint32_t wrap = (1u << bits) - 1;
    uint32_t s = word_slot(word, bits);
    for (uint32_t i = 0; i <= wrap; ++i) {
        const uint32_t k = atomicCAS(&table[s].x, kNoWord, word);
        if (k == kNoWord || k == word) {
            atomicOr(&table[s].y, mask);
            return;
        }
        s = (s + 1) & wrap;
    }
}

// Mask of `word` in the table, 0 if absent.
__device__ __forceinline__ uint32_t table_mask(const uint2* table, uint32_t bits, uint32_t word) {
    const uint32_t wrap = (1u << bits) - 1;
    uint32_t s = word_slot(word, bits);
    for (uint32_t i = 0; i <= wrap; ++i) {
        const uint2 e = table[s];
        if (e.x == word) return e.y;
        if (e.x == kNoWord) return 0u;
        s = (s + 1) & wrap;
    }
    return 0u;
}

// ---------------------------------------------------------------- word lists

// A vertex of one entry is in no triangle: it has no list, and is in none. Such
// vertices rank last, from `limit` on (a star of 2 M leaves: triangles 0.91 -> 0.12 ms,
// its first k-truss 4.2 -> 0.49).
//
// Whether a vertex that ranks x is in the list of its neighbour of rank `own`: below
// it, or any (but itself: a self-loop is in no triangle).
__device__ __forceinline__ bool in_list(uint32_t x, uint32_t own, uint32_t limit, bool full) {
    return full ? x != own && x < limit : x < own;
}

// Room for a list of n words: it starts on 16 bytes and is padded to an even
// length with an empty word, so that the count can read two words at a time.
__device__ __forceinline__ unsigned long long take_words(uint2* words, unsigned long long* cursor, uint32_t n) {
    const unsigned long long at = atomicAdd(cursor, static_cast<unsigned long long>(n + (n & 1)));
    if (n & 1) words[at + n] = make_uint2(kNoWord, 0u);
    return at;
}

// Rows of at most kWarpRow neighbours: up to 32 by matching equal words across
// the lanes, longer ones through a hash table of the warp. A list's place
// comes from a shared cursor (the order of the lists has no meaning).
__global__ void __launch_bounds__(kTwThreads) tw_build_warp_kernel(const uint32_t* __restrict__ offsets,
                                                                   const uint32_t* __restrict__ targets,
                                                                   const uint32_t* __restrict__ rank, uint32_t V,
                                                                   const uint32_t* __restrict__ limit_of, bool full,
                                                                   uint32_t turn, uint2* __restrict__ lists,
                                                                   uint2* __restrict__ words,
                                                                   unsigned long long* __restrict__ cursor) {
    __shared__ uint2 s_table[kTwWarps][1u << kWarpBits];
    __shared__ uint4 s_rows[kTwWarps][32];
    const unsigned lane = lane_id();
    uint2* table = s_table[threadIdx.x >> 5];
    const uint32_t limit = *limit_of;
    const uint64_t warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    // `turn` vertices per warp turn (up to 32; fewer on a small graph, so that
    // every warp has some).
    for (uint64_t v0 = ((static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * turn; v0 < V;
         v0 += warps * turn) {
        const uint64_t my = v0 + lane;
        uint32_t s = 0, d = 0, r = 0;
        if (my < V && lane < turn) {
            s = offsets[my];
            d = offsets[my + 1] - s;
            r = rank[my];
            if (d < 2) {
                d = 0;
                lists[my] = make_uint2(0u, 0u);
            }
        }
        // Rows of up to 32 neighbours: 8, 16 or 32 lanes each, so 4, 2 or 1 rows
        // per step; equal words of a row find each other by a match over (row,
        // word), and the step's rows take their room with one atomic.
#pragma unroll
        for (uint32_t log_size = 3; log_size <= 5; ++log_size) {
            const uint32_t size = 1u << log_size, groups = 32u >> log_size;
            const unsigned rows = __ballot_sync(kFullMask, d > (log_size == 3 ? 0u : size / 2) && d <= size);
            if (rows == 0) continue;
            __syncwarp();
            if ((rows >> lane) & 1u) s_rows[threadIdx.x >> 5][__popc(rows & ((1u << lane) - 1))] = make_uint4(s, d, r, lane);
            __syncwarp();
            const uint32_t n_rows = __popc(rows), group = lane >> log_size, at = lane & (size - 1);
            const unsigned mates = (size == 32 ? kFullMask : ((1u << size) - 1) << (group * size));
            for (uint32_t b = 0; b < n_rows; b += groups) {
                const bool real = b + group < n_rows;
                const uint4 row = real ? s_rows[threadIdx.x >> 5][b + group] : make_uint4(0u, 0u, 0u, 0u);
                const uint32_t x = at < row.y ? __ldg(rank + __ldg(targets + row.x + at)) : kNoWord;
                const bool keep = x != kNoWord && in_list(x, row.z, limit, full);
                // Words are below 2^27: the row's group goes above.
                const unsigned peers = __match_any_sync(kFullMask, keep ? x >> 5 | group << 27 : kNoWord);
                const uint32_t mask = __reduce_or_sync(peers, keep ? 1u << (x & 31) : 0u);
                const bool first = keep && lane == static_cast<unsigned>(__ffs(peers) - 1);
                const unsigned firsts = __ballot_sync(kFullMask, first);
                const uint32_t n = __popc(firsts & mates), padded = n + (n & 1);
                const uint32_t upto = warp_inclusive_scan(at == 0 ? padded : 0u);
                const uint32_t all = __shfl_sync(kFullMask, upto, 31);
                unsigned long long base = 0;
                if (all) {
                    if (lane == 0) base = atomicAdd(cursor, static_cast<unsigned long long>(all));
                    base = __shfl_sync(kFullMask, base, 0) + upto - padded;
                    if (first) words[base + __popc(firsts & mates & ((1u << lane) - 1))] = make_uint2(x >> 5, mask);
                    if (at == 0 && (n & 1)) words[base + n] = make_uint2(kNoWord, 0u);
                }
                if (real && at == 0) lists[v0 + row.w] = make_uint2(static_cast<uint32_t>(base / 2), n);
            }
        }
        unsigned todo = __ballot_sync(kFullMask, d > 32 && d <= kWarpRow);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t rs = __shfl_sync(kFullMask, s, l), rd = __shfl_sync(kFullMask, d, l);
            const uint32_t ru = __shfl_sync(kFullMask, r, l);
            uint32_t n = 0;
            unsigned long long at = 0;
            for (uint32_t k = lane; k < (1u << kWarpBits); k += 32) table[k] = make_uint2(kNoWord, 0u);
            __syncwarp();
            for (uint32_t k = lane; k < rd; k += 32) {
                const uint32_t x = __ldg(rank + __ldg(targets + rs + k));
                if (in_list(x, ru, limit, full)) table_or(table, kWarpBits, x >> 5, 1u << (x & 31));
            }
            __syncwarp();
            for (uint32_t k = lane; k < (1u << kWarpBits); k += 32)
                n += __popc(__ballot_sync(kFullMask, table[k].x != kNoWord));
            if (n) {
                if (lane == 0) at = take_words(words, cursor, n);
                at = __shfl_sync(kFullMask, at, 0);
                unsigned long long to = at;
                for (uint32_t k = lane; k < (1u << kWarpBits); k += 32) {
                    const uint2 e = table[k];
                    const unsigned has = __ballot_sync(kFullMask, e.x != kNoWord);
                    if (e.x != kNoWord) words[to + __popc(has & ((1u << lane) - 1))] = e;
                    to += __popc(has);
                }
            }
            __syncwarp();
            if (lane == 0) lists[v0 + l] = make_uint2(static_cast<uint32_t>(at / 2), n);
        }
    }
}

// Appends, per warp, the vertices with `take` set.
__device__ __forceinline__ void append_vertex(bool take, uint32_t v, uint32_t* __restrict__ list,
                                              uint32_t* __restrict__ count) {
    const unsigned mask = __ballot_sync(kFullMask, take);
    if (mask == 0) return;
    uint32_t at = 0;
    const int leader = __ffs(mask) - 1;
    if (lane_id() == static_cast<unsigned>(leader)) at = atomicAdd(count, static_cast<uint32_t>(__popc(mask)));
    at = __shfl_sync(kFullMask, at, leader);
    if (take) list[at + __popc(mask & ((1u << lane_id()) - 1))] = v;
}

__global__ void tw_long_rows_kernel(const uint32_t* __restrict__ offsets, uint32_t V, uint32_t* __restrict__ list,
                                    uint32_t* __restrict__ count) {
    for (uint64_t b = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) & ~31ull; b < V;
         b += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t v = b + lane_id();
        append_vertex(v < V && offsets[v + 1] - offsets[v] > kWarpRow, static_cast<uint32_t>(v), list, count);
    }
}

// Longer rows, a CTA each: the ranks of the list are set in a bitmap,
// bitmap_words * 32 of them at a time, and its non-zero words written out. Two
// sweeps of the row where it has more than one window: the first counts. A row is
// read kRowLoads entries per thread at a time (one at a time, a hub of 2 M entries
// took 5 ms). The longest rows are those of the lowest ranks, and the vertices that
// rank below them few: where there are kSearchRatio times more entries than those,
// they are looked up in the row instead (triangles of that star 5.8 -> 0.9 ms).
constexpr int kRowLoads = 8;
constexpr uint32_t kSearchRatio = 32;

__global__ void __launch_bounds__(1024) tw_build_cta_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, const uint32_t* __restrict__ rank,
    const uint32_t* __restrict__ at_rank, const uint32_t* __restrict__ limit, bool full, uint32_t bitmap_words,
    const uint32_t* __restrict__ rows,
    const uint32_t* __restrict__ n_rows, uint32_t* __restrict__ next, uint2* __restrict__ lists,
    uint2* __restrict__ words, unsigned long long* __restrict__ cursor) {
    extern __shared__ uint32_t s_bits[];
    __shared__ uint32_t s_item, s_total, s_at;
    __shared__ unsigned long long s_base;
    const unsigned lane = lane_id();
    const uint32_t window = bitmap_words * 32;
    for (uint32_t k = threadIdx.x; k < bitmap_words; k += blockDim.x) s_bits[k] = 0;
    const uint32_t n = *n_rows;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            s_item = atomicAdd(next, 1u);
            s_total = 0;
            s_at = 0;
        }
        __syncthreads();
        if (s_item >= n) break;
        const uint32_t u = rows[s_item];
        const uint32_t s = offsets[u], e = offsets[u + 1], r = rank[u];
        const uint32_t end = full ? *limit : r;  // of the ranks in the list
        const uint32_t windows = static_cast<uint32_t>(ceil_div_u64(end, window));
        for (uint32_t sweep = windows > 1 ? 0 : 1; sweep < 2; ++sweep) {
            for (uint32_t w = 0; w < max(windows, 1u); ++w) {
                const uint32_t lo = w * window, hi = min(end - lo, window) + lo;
                if ((e - s) / kSearchRatio > end) {
                    for (uint32_t x = lo + threadIdx.x; x < hi; x += blockDim.x) {
                        const uint32_t v = __ldg(at_rank + x), p = lower_bound_u32(targets, s, e, v);
                        if (p < e && targets[p] == v && x != r) atomicOr(s_bits + ((x - lo) >> 5), 1u << (x & 31));
                    }
                } else {
                    for (uint64_t j = static_cast<uint64_t>(s) + threadIdx.x; j < e; j += kRowLoads * blockDim.x) {
                        uint32_t x[kRowLoads];
#pragma unroll
                        for (int q = 0; q < kRowLoads; ++q) {
                            const uint64_t i = j + static_cast<uint64_t>(q) * blockDim.x;
                            x[q] = ld_nc_if(i < e, targets + i, 0u);
                        }
#pragma unroll
                        for (int q = 0; q < kRowLoads; ++q)
                            x[q] = ld_nc_if(j + static_cast<uint64_t>(q) * blockDim.x < e, rank + x[q], r);
#pragma unroll
                        for (int q = 0; q < kRowLoads; ++q)
                            if (x[q] >= lo && x[q] < hi && x[q] != r)
                                atomicOr(s_bits + ((x[q] - lo) >> 5), 1u << (x[q] & 31));
                    }
                }
                __syncthreads();
                const uint32_t used = (hi - lo + 31) / 32;
                if (windows <= 1 || sweep == 0) {
                    uint32_t mine = 0;
                    for (uint32_t k = threadIdx.x; k < used; k += blockDim.x) {
                        mine += s_bits[k] != 0 ? 1u : 0u;
                        if (windows > 1) s_bits[k] = 0;
                    }
                    mine = warp_sum(mine);
                    if (lane == 0 && mine) atomicAdd(&s_total, mine);
                }
                __syncthreads();
                if (sweep == 1) {
                    if (w == 0) {
                        if (threadIdx.x == 0) {
                            s_base = s_total ? take_words(words, cursor, s_total) : 0ull;
                            lists[u] = make_uint2(static_cast<uint32_t>(s_base / 2), s_total);
                        }
                        __syncthreads();
                    }
                    for (uint32_t k0 = threadIdx.x & ~31u; k0 < used; k0 += blockDim.x) {
                        const uint32_t k = k0 + lane;
                        const uint32_t m = k < used ? s_bits[k] : 0u;
                        const unsigned has = __ballot_sync(kFullMask, m != 0);
                        if (has == 0) continue;
                        uint32_t at = 0;
                        if (lane == 0) at = atomicAdd(&s_at, static_cast<uint32_t>(__popc(has)));
                        at = __shfl_sync(kFullMask, at, 0);
                        if (m) {
                            words[s_base + at + __popc(has & ((1u << lane) - 1))] = make_uint2((lo >> 5) + k, m);
                            s_bits[k] = 0;
                        }
                    }
                }
                __syncthreads();
            }
        }
    }
}

// First word of a list.
__device__ __forceinline__ const uint2* list_words(const uint2* __restrict__ words, const uint2 l) {
    return words + 2ull * l.x;
}

// ---------------------------------------------------------------- owners

// Vertices with words: to the warp kernel's list, or as (vertex, slice) items
// to the CTA kernel's. A list of one neighbour shares none with that one's, and
// edges between lists of one word belong to the higher rank, which has both ends
// of a triangle's third edge in its own: such a vertex owns nothing (all vertices of
// a forest).
__global__ void tw_owners_kernel(const uint32_t* __restrict__ offsets, const uint2* __restrict__ lists,
                                 const uint2* __restrict__ words, uint32_t V, uint32_t warp_words,
                                 uint32_t* __restrict__ warp_list, uint32_t* __restrict__ warp_count,
                                 uint2* __restrict__ items, uint32_t* __restrict__ item_count) {
    for (uint64_t b = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) & ~31ull; b < V;
         b += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t v = b + lane_id();
        uint32_t n = 0, d = 0;
        if (v < V) {
            const uint2 l = lists[v];
            n = l.y;
            d = offsets[v + 1] - offsets[v];
            if (n == 1 && __popc(__ldg(list_words(words, l)).y) == 1) n = 0;
        }
        const bool alone = n <= warp_words && d <= kWarpOwnerRow;  // a warp's
        append_vertex(n > 0 && alone, static_cast<uint32_t>(v), warp_list, warp_count);
        // One place per warp step: an atomic per vertex on the one counter bounded
        // this kernel (R-MAT 22 262 -> 121 us).
        const uint32_t slices = n > 0 && !alone ? (d + kSlice - 1) / kSlice : 0u;
        const uint32_t upto = warp_inclusive_scan(slices), all = __shfl_sync(kFullMask, upto, 31);
        if (all == 0) continue;
        uint32_t at = 0;
        if (lane_id() == 0) at = atomicAdd(item_count, all);
        at = __shfl_sync(kFullMask, at, 0) + upto - slices;
        for (uint32_t k = 0; k < slices; ++k) items[at + k] = make_uint2(static_cast<uint32_t>(v), k);
    }
}

// ---------------------------------------------------------------- counting

// Two words from word `at` (even) of a list, whose place is kept in units of two
// words.
__device__ __forceinline__ uint4 word_pair(const uint2* __restrict__ words, const uint2 l, uint32_t at) {
    return __ldg(reinterpret_cast<const uint4*>(words) + (l.x + at / 2));
}

// The warp's neighbours in hand: their lists and, for the support, the entries
// whose support their counts are.
template <bool kSupport>
struct ListBox {
    uint2 list[32];
    uint32_t entry[kSupport ? 32 : 1];
};

// Streams the lists l with `take` against mask(word), 2^kLogSize lanes per list
// (a lane reads two words at a time) and kInFlight lists in flight per group of
// lanes; with 32 lanes per list, lists may be longer than the group. The hits
// are summed over all lists (the lane's part is returned), or, with kSupport,
// over the lanes of each list and given to store(entry, sum).
template <uint32_t kLogSize, bool kSupport, class Mask, class Store>
__device__ __forceinline__ uint32_t stream_lists(bool take, const uint2 l, uint32_t entry,
                                                 const uint2* __restrict__ words, ListBox<kSupport>& box, Mask mask,
                                                 Store store) {
    const unsigned lane = lane_id();
    const unsigned taken = __ballot_sync(kFullMask, take);
    if (taken == 0) return 0;
    constexpr uint32_t size = 1u << kLogSize, groups = 32u >> kLogSize;
    const uint32_t count = __popc(taken), group = lane >> kLogSize, at = 2 * (lane & (size - 1));
    __syncwarp();
    if (take) {
        const uint32_t k = __popc(taken & ((1u << lane) - 1));
        box.list[k] = l;
        if constexpr (kSupport) box.entry[k] = entry;
    }
    __syncwarp();
    uint32_t hits = 0;
    auto popcounts = [&](const uint4& p) { return __popc(mask(p.x) & p.y) + __popc(mask(p.z) & p.w); };
    for (uint32_t b = 0; b < count; b += kInFlight * groups) {
        uint2 e[kInFlight];
        uint4 p[kInFlight];
        uint32_t sum[kInFlight];
#pragma unroll
        for (int i = 0; i < kInFlight; ++i) {
            const uint32_t k = b + i * groups + group;
            e[i] = k < count ? box.list[k] : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < kInFlight; ++i)
            p[i] = at < e[i].y ? word_pair(words, e[i], at)
                               : make_uint4(kNoWord, 0u, kNoWord, 0u);
#pragma unroll
        for (int i = 0; i < kInFlight; ++i) {
            if constexpr (kSupport) sum[i] = 0;
            if (at < e[i].y) (kSupport ? sum[i] : hits) += popcounts(p[i]);
        }
        if (kLogSize == 5) {
#pragma unroll
            for (int i = 0; i < kInFlight; ++i) {
                uint32_t k = at + 64;
                for (; k + 64 < e[i].y; k += 128) {
                    const uint4 x = word_pair(words, e[i], k);
                    const uint4 y = word_pair(words, e[i], k + 64);
                    (kSupport ? sum[i] : hits) += popcounts(x);
                    (kSupport ? sum[i] : hits) += popcounts(y);
                }
                if (k < e[i].y) (kSupport ? sum[i] : hits) += popcounts(word_pair(words, e[i], k));
            }
        }
        if constexpr (kSupport) {
#pragma unroll
            for (int i = 0; i < kInFlight; ++i) {
                if (kLogSize == 5) {
                    sum[i] = __reduce_add_sync(kFullMask, sum[i]);
                } else {
#pragma unroll
                    for (uint32_t d = size / 2; d > 0; d /= 2) sum[i] += __shfl_xor_sync(kFullMask, sum[i], d);
                }
                const uint32_t k = b + i * groups + group;
                if (at == 0 && k < count && sum[i]) store(box.entry[k], sum[i]);
            }
        }
    }
    return hits;
}

// Up to 32 neighbours (v per lane, `valid`) of an owner with id u and n words:
// the lists of those it owns the edge to (fewer words, or as many and a smaller
// id; one word each: a lower rank), by length: up to 8 words 4 lanes each, up to 32 words 16, the others 32.
// j: the CSR entry of the neighbour; the support of an edge is kept at its
// entry in the smaller vertex's row.
template <bool kSupport, class Mask, class Store>
__device__ __forceinline__ uint32_t count_neighbours(bool valid, uint32_t j, uint32_t v, uint32_t u, uint32_t n,
                                                     const uint2* __restrict__ lists, const uint2* __restrict__ words,
                                                     const uint32_t* __restrict__ rank, const uint32_t* __restrict__ rev,
                                                     ListBox<kSupport>& box, Mask mask, Store store) {
    const uint2 l = valid ? __ldg(lists + v) : make_uint2(0u, 0u);
    bool below = v < u;
    if (n == 1) below = valid && __ldg(rank + v) < __ldg(rank + u);
    const bool take = l.y > 0 && (l.y < n || (l.y == n && below));
    uint32_t entry = 0;
    if constexpr (kSupport) entry = take ? (u < v ? j : __ldg(rev + j)) : 0u;
    return stream_lists<2, kSupport>(take && l.y <= 8, l, entry, words, box, mask, store) +
           stream_lists<4, kSupport>(take && l.y > 8 && l.y <= 32, l, entry, words, box, mask, store) +
           stream_lists<5, kSupport>(take && l.y > 32, l, entry, words, box, mask, store);
}

// Total, or per owner (a union's graphs are told apart by their owners).
__device__ __forceinline__ void add_owner(uint32_t u, uint32_t hits, unsigned long long* __restrict__ per_vertex,
                                          unsigned long long& total) {
    if (per_vertex) {
        const uint32_t sum = __reduce_add_sync(kFullMask, hits);
        if (lane_id() == 0 && sum) atomicAdd(per_vertex + u, static_cast<unsigned long long>(sum));
    } else {
        total += hits;
    }
}

// What the kernel counts: triangles, in total or per owner, or the support of
// every edge (full lists).
struct WordCount {
    unsigned long long* total;
    unsigned long long* per_vertex;
    uint32_t V;
    uint32_t bitmap_words;  // of the support's dynamic shared array
    const uint32_t* rev;
    uint32_t* support;
};

// Blocks take the CTA items first, then their warps take the warp owners: the
// end of the one fills the idle warps with the other. Everyone's first turn is its
// own number and only what is beyond those is handed out by counters: on a small graph
// the atomics on them were a third of a count (8 graphs of 1,000 vertices 27 -> 21 us).
template <bool kSupport, int kThreads, int kCtasPerSm>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) tw_count_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, const uint32_t* __restrict__ rank,
    const uint2* __restrict__ lists, const uint2* __restrict__ words, const uint2* __restrict__ items,
    const uint32_t* __restrict__ owners, const uint32_t* __restrict__ counts, uint32_t* __restrict__ next,
    uint32_t batch, const WordCount out) {
    // Words as a bitmap, pairs of words as a table: 8-byte accesses.
    __shared__ __align__(16) uint32_t s_fixed[kSupport ? 1 : kBitmapWords];
    extern __shared__ __align__(16) uint32_t s_dynamic[];
    __shared__ ListBox<kSupport> s_box[kThreads / 32];
    __shared__ uint32_t s_item, s_chunk;
    uint32_t* s_bits = kSupport ? s_dynamic : s_fixed;
    const uint32_t bitmap_words = kSupport ? out.bitmap_words : kBitmapWords;
    uint2* table = reinterpret_cast<uint2*>(s_bits);
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t n_items = counts[3], n_owners = counts[2];
    unsigned long long sum = 0;
    if (n_items)
        for (uint32_t k = threadIdx.x; k < bitmap_words; k += kThreads) s_bits[k] = 0;
    for (uint32_t turn = 0;; ++turn) {
        __syncthreads();
        if (threadIdx.x == 0)
            s_item = turn == 0 ? blockIdx.x : gridDim.x < n_items ? gridDim.x + atomicAdd(next, 1u) : n_items;
        __syncthreads();
        if (s_item >= n_items) break;
        const uint2 item = items[s_item];
        const uint32_t u = item.x;
        const uint2 own = __ldg(lists + u);
        const uint32_t s = offsets[u] + item.y * kSlice, e = s + min(kSlice, offsets[u + 1] - s);
        const uint32_t end = kSupport ? out.V : rank[u];  // of the ranks in the owner's list
        const uint32_t window = bitmap_words * 32;
        const bool hash = end > window && own.y <= kHashWords;
        const uint32_t windows = hash ? 1u : static_cast<uint32_t>(ceil_div_u64(end, window));
        uint32_t hits = 0;
        for (uint32_t win = 0; win < windows; ++win) {
            const uint32_t lo = win * bitmap_words;
            if (hash) {
                for (uint32_t k = threadIdx.x; k < (1u << kHashBits); k += kThreads)
                    table[k] = make_uint2(kNoWord, 0u);
                __syncthreads();
            }
            for (uint32_t k = threadIdx.x; k < own.y; k += kThreads) {
                const uint2 w = __ldg(list_words(words, own) + k);
                if (hash) table_or(table, kHashBits, w.x, w.y);
                else if (w.x - lo < bitmap_words) s_bits[w.x - lo] = w.y;  // the words of a list are distinct
            }
            if (threadIdx.x == 0) s_chunk = 0;
            __syncthreads();
            // A later window adds to what the block stored before the barrier.
            auto store = [&](uint32_t entry, uint32_t h) { out.support[entry] = win ? out.support[entry] + h : h; };
            while (true) {
                uint32_t c = 0;
                if (lane == 0) c = atomicAdd(&s_chunk, 32u);
                c = __shfl_sync(kFullMask, c, 0);
                if (c >= e - s) break;
                const bool valid = e - s - c > lane;
                const uint32_t j = s + c + lane;
                const uint32_t v = valid ? ld_stream(targets + j) : 0u;
                if (hash)
                    hits += count_neighbours<kSupport>(
                        valid, j, v, u, own.y, lists, words, rank, out.rev, s_box[warp],
                        [&](uint32_t w) { return table_mask(table, kHashBits, w); }, store);
                else
                    hits += count_neighbours<kSupport>(
                        valid, j, v, u, own.y, lists, words, rank, out.rev, s_box[warp],
                        [&](uint32_t w) { return w - lo < bitmap_words ? s_bits[w - lo] : 0u; }, store);
            }
            __syncthreads();
            if (hash) {
                for (uint32_t k = threadIdx.x; k < (2u << kHashBits); k += kThreads) s_bits[k] = 0;
            } else {
                for (uint32_t k = threadIdx.x; k < own.y; k += kThreads) {
                    const uint32_t w = __ldg(list_words(words, own) + k).x;
                    if (w - lo < bitmap_words) s_bits[w - lo] = 0;
                }
            }
            if (win + 1 < windows) __syncthreads();
        }
        if (!kSupport) add_owner(u, hits, out.per_vertex, sum);
    }
    table += warp << kWarpBits;  // the warps' own tables from here on (after the loop's block barrier)
    auto store = [&](uint32_t entry, uint32_t h) { out.support[entry] = h; };
    const uint32_t own_turns = gridDim.x * (kThreads / 32) * batch;
    for (uint32_t base = (blockIdx.x * (kThreads / 32) + warp) * batch; base < n_owners;) {
        const uint32_t last = min(base + batch, n_owners);
        for (uint32_t h = base; h < last; ++h) {
            const uint32_t u = owners[h];
            const uint2 own = __ldg(lists + u);
            const uint32_t s = offsets[u], e = offsets[u + 1];
            uint32_t bits = 5;  // load at most 3/8
            while (bits < kWarpBits && (1u << bits) * 3 < own.y * 8) ++bits;
            __syncwarp();
            for (uint32_t k = lane; k < (1u << bits); k += 32) table[k] = make_uint2(kNoWord, 0u);
            __syncwarp();
            for (uint32_t k = lane; k < own.y; k += 32) {
                const uint2 w = __ldg(list_words(words, own) + k);
                table_or(table, bits, w.x, w.y);
            }
            __syncwarp();
            uint32_t hits = 0;
            walk_entries(s, e, 32, [&](uint32_t o) {
                const bool valid = e - s - o > lane;
                const uint32_t j = s + o + lane;
                const uint32_t v = valid ? ld_stream(targets + j) : 0u;
                hits += count_neighbours<kSupport>(
                    valid, j, v, u, own.y, lists, words, rank, out.rev, s_box[warp],
                    [&](uint32_t w) { return table_mask(table, bits, w); }, store);
            });
            if (!kSupport) add_owner(u, hits, out.per_vertex, sum);
        }
        if (own_turns >= n_owners) break;
        if (lane == 0) base = own_turns + atomicAdd(next + 1, batch);
        base = __shfl_sync(kFullMask, base, 0);
    }
    if (!kSupport) {
        sum = warp_sum(sum);
        if (lane == 0 && sum) atomicAdd(out.total, sum);
    }
}

}  // namespace

// ---------------------------------------------------------------- host

namespace {

// Bitmap of the full lists' ranks: all of them, or as many as fit an SM.
uint32_t support_bitmap_words(uint32_t V) {
    // Room for the warps' tables too (1024 threads: 32 tables).
    const uint64_t words = ceil_div_u64(V, 32);
    const uint64_t tables = words * sizeof(uint32_t) <= kBitmap256 ? kBitmapWords : kMaxTableWords;
    return static_cast<uint32_t>(std::min<uint64_t>(std::max(words, tables), kMaxBitmapWords));
}

}  // namespace

Error build_word_lists(GraphImpl& g, bool full, WordLists* w, WordListSizes* size) {
    DeviceImpl& dev = *g.dev;
    const uint32_t V = g.num_nodes, E = g.num_edges;
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    DeviceBuffer<uint32_t> at_rank;  // [V] = the first rank of one entry or none
    GCU_TRY(degree_class_order(dev, g.offsets.ptr, V, &w->rank, &at_rank));
    const uint32_t* limit = at_rank.ptr + V;
    GCU_TRY(w->lists.allocate(dev, V));
    // An edge's ranks are kept at one end, or at both: E / 2 or E words at most,
    // and a padding word per list (lists without words take no room).
    const uint64_t kept = full ? E : E / 2;
    const uint64_t room = kept + std::min<uint64_t>(kept, V);
    GCU_TRY(w->words.allocate(dev, std::max<uint64_t>(room, 1)));
    GCU_TRY(w->warp_owners.allocate(dev, V));
    // counters: [0] long rows, [1] next long row, [2] warp owners, [3] CTA items
    GCU_TRY(w->counts.allocate(dev, 4));
    DeviceBuffer<unsigned long long> cursor;
    GCU_TRY(cursor.allocate(dev, 1));
    GCU_CUDA(cudaMemsetAsync(w->counts.ptr, 0, 4 * sizeof(uint32_t), dev.stream), "memset");
    GCU_CUDA(cudaMemsetAsync(cursor.ptr, 0, sizeof(unsigned long long), dev.stream), "memset");
    const unsigned vgrid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(V, 256), cap)));
    uint32_t turn = 32;
    while (turn > 4 && V / turn < static_cast<uint64_t>(dev.sm_count) * 8 * kTwWarps) turn /= 2;
    const unsigned wgrid = static_cast<unsigned>(
        std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(V, static_cast<uint64_t>(turn) * kTwWarps), cap)));
    GCU_LAUNCH(dev, "tw_build_warp", tw_build_warp_kernel, wgrid, kTwThreads, 0, g.offsets.ptr, g.targets.ptr,
               w->rank.ptr, V, limit, full, turn, w->lists.ptr, w->words.ptr, cursor.ptr);
    // The owner list is free until the owners are known: the long rows use it.
    GCU_LAUNCH(dev, "tw_long_rows", tw_long_rows_kernel, vgrid, 256, 0, g.offsets.ptr, V, w->warp_owners.ptr,
               w->counts.ptr);
    // Full lists: all ranks in one window while the bitmap fits an SM.
    const uint32_t bitmap_words = full ? support_bitmap_words(V) : kBitmapWords;
    const unsigned threads = bitmap_words * sizeof(uint32_t) > kBitmap512 ? 1024u : kTwThreads;
    const size_t smem = sizeof(uint32_t) * bitmap_words;
    GCU_CUDA(cudaFuncSetAttribute(tw_build_cta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(sizeof(uint32_t) * kMaxBitmapWords)),
             "cudaFuncSetAttribute");
    const unsigned resident = static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>(7, kSmemPerSm / (smem + 2048))));
    const unsigned cgrid = static_cast<unsigned>(
        std::max<uint64_t>(1, std::min<uint64_t>(E / kWarpRow, static_cast<uint64_t>(dev.sm_count) * resident)));
    GCU_LAUNCH(dev, "tw_build_cta", tw_build_cta_kernel, cgrid, threads, smem, g.offsets.ptr, g.targets.ptr,
               w->rank.ptr, at_rank.ptr, limit, full, bitmap_words, w->warp_owners.ptr, w->counts.ptr, w->counts.ptr + 1, w->lists.ptr,
               w->words.ptr, cursor.ptr);
    // Items: at most one per kSlice entries plus one per vertex with more words,
    // so more neighbours, than a warp owner.
    const uint32_t warp_words = !full && V < kSmallGraph ? kWarpWordsSmall : kWarpWords;
    w->max_items = E / kSlice + E / warp_words + 1;
    GCU_TRY(w->items.allocate(dev, w->max_items));
    GCU_LAUNCH(dev, "tw_owners", tw_owners_kernel, vgrid, 256, 0, g.offsets.ptr, w->lists.ptr, w->words.ptr, V, warp_words,
               w->warp_owners.ptr, w->counts.ptr + 2, w->items.ptr, w->counts.ptr + 3);
    if (size) {
        uint32_t counts[2];
        GCU_CUDA(cudaMemcpyAsync(&size->words, cursor.ptr, sizeof(uint64_t), cudaMemcpyDeviceToHost, dev.stream), "copy");
        GCU_CUDA(cudaMemcpyAsync(counts, w->counts.ptr + 2, sizeof(counts), cudaMemcpyDeviceToHost, dev.stream), "copy");
        GCU_TRY(dev.sync());
        size->owners = static_cast<uint64_t>(counts[0]) + counts[1];
    }
    return ok();
}

namespace {

// kMaxSmem: the most dynamic shared memory that a graph of this form asks for. The
// kernel's limit is set to it, not to this graph's need: it belongs to the kernel,
// and another thread may launch it on a graph with another need.
template <bool kSupport, int kThreads, int kCtasPerSm, size_t kMaxSmem>
Error launch_count(GraphImpl& g, const WordLists& w, uint32_t* next, const WordCount& out) {
    DeviceImpl& dev = *g.dev;
    constexpr int kWarps = kThreads / 32;
    const size_t smem = sizeof(uint32_t) * out.bitmap_words;
    const auto kernel = tw_count_kernel<kSupport, kThreads, kCtasPerSm>;
    if (kMaxSmem)
        GCU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxSmem)),
                 "cudaFuncSetAttribute");
    GCU_CUDA(cudaMemsetAsync(next, 0, 2 * sizeof(uint32_t), dev.stream), "memset");
    const uint64_t want = std::max<uint64_t>(w.max_items, ceil_div_u64(g.num_nodes, kWarps));
    const unsigned grid = static_cast<unsigned>(
        std::max<uint64_t>(1, std::min<uint64_t>(want, static_cast<uint64_t>(dev.sm_count) * kCtasPerSm)));
    // Owners per handout: several turns per warp, or one at a time on a small graph.
    const uint32_t batch = static_cast<uint32_t>(
        std::max<uint64_t>(1, std::min<uint64_t>(8, g.num_nodes / (static_cast<uint64_t>(grid) * kWarps * 8))));
    GCU_LAUNCH(dev, kSupport ? "tw_support" : "tw_count", kernel, grid, kThreads, smem, g.offsets.ptr, g.targets.ptr,
               w.rank.ptr, w.lists.ptr, w.words.ptr, w.items.ptr, w.warp_owners.ptr, w.counts.ptr, next, batch, out);
    return ok();
}

}  // namespace

Error count_words(GraphImpl& g, const WordLists& w, uint32_t* next, unsigned long long* total,
                  unsigned long long* per_vertex) {
    return launch_count<false, kCountThreads, kCountCtasPerSm, 0>(
        g, w, next, WordCount{total, per_vertex, g.num_nodes, 0, nullptr, nullptr});
}

Error edge_support(GraphImpl& g, const uint32_t* rev, uint32_t* support) {
    DeviceImpl& dev = *g.dev;
    WordLists w;
    GCU_TRY(build_word_lists(g, true, &w));
    DeviceBuffer<uint32_t> next;
    GCU_TRY(next.allocate(dev, 2));
    WordCount out{nullptr, nullptr, g.num_nodes, support_bitmap_words(g.num_nodes), rev, support};
    const size_t bytes = sizeof(uint32_t) * out.bitmap_words;
    if (bytes <= kBitmap128) GCU_TRY((launch_count<true, 128, 12, kBitmap128>(g, w, next.ptr, out)));
    else if (bytes <= kBitmap256) GCU_TRY((launch_count<true, 256, 6, kBitmap256>(g, w, next.ptr, out)));
    else if (bytes <= kBitmap512) GCU_TRY((launch_count<true, 512, 3, kBitmap512>(g, w, next.ptr, out)));
    else GCU_TRY((launch_count<true, 1024, 1, sizeof(uint32_t) * kMaxBitmapWords>(g, w, next.ptr, out)));
    return dev.sync();  // the lists are freed on return
}

}  // namespace gcu

// k-truss by synchronous peeling.
//
// Reference: crates/grafeo-cuda-algos/src/k_truss.rs:42-161 and
// kernels/k_truss.cu:46-124. Each reference round computes, for every live CSR
// entry u -> v with v > u, support = |live N(u) ∩ live N(v)| (entry-level
// liveness, so in the first round a live self-loop at u or v counts as a
// common neighbour, as the reference's merge of the raw lists does), copies it
// to the live reverse entry v -> u, and then removes every live entry whose
// support is below k - 2. Rounds repeat until one removes nothing; their count
// is the reference's `iterations`. Two paths give exactly the same removed
// sets round by round, hence the same edges and round count:
//
//  * Symmetric CSR (every graph exported from Grafeo): the support of every
//    undirected edge is its triangle count, found once as the popcount of its
//    ends' neighbour bits (edge_support, tri_words.cu); round 1 adds one for a
//    self-loop at either end. After a
//    round removes a set R of edges, each triangle with an edge in R that was
//    alive at the start of the round is destroyed once (credited to its
//    removed edge with the smallest id) and its surviving edges lose one
//    support, so the supports stay exact for the next round without
//    recomputing them. Work per round is proportional to the edges removed.
//  * Any other CSR: the reference's per-entry rules with all supports
//    recomputed each round (a warp per entry, binary-search intersection).
//
// Both paths use a reverse-entry index instead of the reference's linear scan
// of N(v), and compact the result edge list on the device in CSR order (the
// reference copies removed/offsets/targets back and loops on the host).
#include <algorithm>

#include "device_common.cuh"
#include "gcu_internal.h"

namespace gcu {

constexpr uint32_t kNone = 0xFFFFFFFFu;

// src[j] = row of entry j.
__global__ void __launch_bounds__(256) kt_rows_kernel(const uint32_t* __restrict__ offsets, uint32_t V, uint32_t E,
                                                      uint32_t* __restrict__ src) {
    for_each_entry<256, 4>(offsets, V, E, [&](uint32_t j, uint32_t row) { src[j] = row; });
}

// rev[j] = index of entry v -> u for entry j = u -> v, or kNone.
__global__ void kt_reverse_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets,
                                  const uint32_t* __restrict__ src, uint32_t E, uint32_t* __restrict__ rev) {
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < E;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t u = src[j], v = targets[j];
        const uint32_t s = offsets[v], e = offsets[v + 1];
        const uint32_t p = lower_bound_u32(targets, s, e, u);
        rev[j] = (p < e && targets[p] == u) ? p : kNone;
    }
}

// The same for a symmetric CSR, both entries of an edge at once: the one in the
// longer list (ties: the larger vertex) searches the shorter list for the other
// (R-MAT 18: 233 -> 125 us against a search per entry).
__global__ void __launch_bounds__(256) kt_pairs_kernel(const uint32_t* __restrict__ offsets,
                                                       const uint32_t* __restrict__ targets,
                                                       const uint32_t* __restrict__ src, uint32_t E,
                                                       uint32_t* __restrict__ rev) {
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < E;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t u = src[j], v = targets[j];
        const uint32_t s = offsets[v], e = offsets[v + 1];
        const uint32_t du = offsets[u + 1] - offsets[u], dv = e - s;
        if (du < dv || (du == dv && u < v)) continue;
        const uint32_t p = lower_bound_u32(targets, s, e, u);
        rev[j] = p;  // u == v: a self-loop's is j itself
        rev[p] = static_cast<uint32_t>(j);
    }
}

// One warp per live entry u -> v with v > u (32 candidate entries per step).
__global__ void __launch_bounds__(256) kt_support_kernel(const uint32_t* __restrict__ offsets,
                                                         const uint32_t* __restrict__ targets,
                                                         const uint32_t* __restrict__ src,
                                                         const uint32_t* __restrict__ rev,
                                                         const uint8_t* __restrict__ live, uint32_t E,
                                                         uint32_t* __restrict__ support) {
    const unsigned lane = lane_id();
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t base = warp * 32; base < E; base += nwarps * 32) {
        const uint64_t j = base + lane;
        uint32_t u = 0, v = 0;
        bool todo = false;
        if (j < E && live[j]) {
            u = src[j];
            v = targets[j];
            todo = v > u;
        }
        unsigned pending = __ballot_sync(kFullMask, todo);
        while (pending) {
            const int l = __ffs(pending) - 1;
            pending &= pending - 1;
            const uint32_t eu = __shfl_sync(kFullMask, u, l), ev = __shfl_sync(kFullMask, v, l);
            uint32_t as = offsets[eu], ae = offsets[eu + 1], bs = offsets[ev], be = offsets[ev + 1];
            if (ae - as > be - bs) {
                uint32_t t = as; as = bs; bs = t;
                t = ae; ae = be; be = t;
            }
            uint32_t hits = 0;
            walk_entries(as, ae, 32, [&](uint32_t o) {
                if (ae - as - o <= lane || !live[as + o + lane]) return;
                const uint32_t x = targets[as + o + lane];
                const uint32_t p = lower_bound_u32(targets, bs, be, x);
                if (p < be && targets[p] == x && live[p]) ++hits;
            });
            hits = warp_sum(hits);
            if (lane == 0) {
                const uint64_t ej = base + l;
                support[ej] = hits;
                const uint32_t r = rev[ej];
                if (r != kNone && live[r]) support[r] = hits;
            }
        }
    }
}

__global__ void kt_filter_kernel(const uint32_t* __restrict__ support, uint8_t* __restrict__ live, uint32_t E,
                                 uint32_t threshold, uint32_t* __restrict__ removed) {
    uint32_t mine = 0;
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < E;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        if (live[j] && support[j] < threshold) {
            live[j] = 0;
            ++mine;
        }
    }
    mine = warp_sum(mine);
    if (lane_id() == 0 && mine) atomicAdd(removed, mine);
}

struct LiveFlag {
    const uint8_t* live;
    __device__ __forceinline__ bool operator()(uint64_t j) const { return live[j] != 0; }
};
struct RoundState {
    const uint32_t* state;  // 0 = alive, r = removed in round r
    __device__ __forceinline__ bool operator()(uint64_t j) const { return state[j] == 0; }
};

template <class Alive>
__global__ void kt_flag_kernel(const uint32_t* __restrict__ targets, const uint32_t* __restrict__ src, Alive alive,
                               uint32_t E, uint32_t* __restrict__ flag) {
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < E;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        flag[j] = (targets[j] > src[j] && alive(j)) ? 1u : 0u;
    }
}

template <class Alive>
__global__ void kt_emit_kernel(const uint32_t* __restrict__ targets, const uint32_t* __restrict__ src, Alive alive,
                               uint32_t E, const uint32_t* __restrict__ pos, uint2* __restrict__ out) {
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < E;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t u = src[j], v = targets[j];
        if (v > u && alive(j)) out[pos[j]] = make_uint2(u, v);
    }
}

// ---------------------------------------------------------------- symmetric CSR: incremental peeling

// loop[u] = 1 for every vertex with a self-loop entry; counts them in *loops.
__global__ void kt_loops_kernel(const uint32_t* __restrict__ targets, const uint32_t* __restrict__ src, uint32_t E,
                                uint8_t* __restrict__ loop, uint32_t* __restrict__ loops) {
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < E;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t u = src[j];
        if (targets[j] == u) {
            loop[u] = 1;
            atomicAdd(loops, 1u);
        }
    }
}

constexpr int kFilterLoads = 4;

// Round r: every alive u < v entry whose support is below the threshold is
// removed (state = r) and listed. With `loop` in round 1 a self-loop at either
// end adds one to the support, as the reference's merge of the raw lists
// does.
__global__ void kt_round_filter_kernel(const uint32_t* __restrict__ targets, const uint32_t* __restrict__ src,
                                       const uint8_t* __restrict__ loop, const uint32_t* __restrict__ support,
                                       uint32_t* __restrict__ state, uint32_t E, uint32_t threshold, uint32_t round,
                                       uint32_t* __restrict__ removed, uint32_t* __restrict__ removed_count) {
    const unsigned lane = lane_id();
    const uint64_t step = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t base = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) & ~31ull; base < E;
         base += kFilterLoads * step) {
        // kFilterLoads entries per lane in flight, and one place in the list for all.
        unsigned taken[kFilterLoads];
        uint32_t total = 0;
#pragma unroll
        for (int q = 0; q < kFilterLoads; ++q) {
            const uint64_t j = base + q * step + lane;
            bool take = false;
            if (j < E) {
                const uint32_t alive = state[j], u = src[j], v = targets[j];
                uint32_t s = support[j];
                if (loop && round == 1) s += loop[u] + loop[v];
                take = alive == 0 && v > u && s < threshold;
            }
            taken[q] = __ballot_sync(kFullMask, take);
            total += __popc(taken[q]);
        }
        if (total == 0) continue;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(removed_count, total);
        at = __shfl_sync(kFullMask, at, 0);
#pragma unroll
        for (int q = 0; q < kFilterLoads; ++q) {
            const uint32_t j = static_cast<uint32_t>(base + q * step + lane);
            if ((taken[q] >> lane) & 1u) {
                state[j] = round;
                removed[at + __popc(taken[q] & ((1u << lane) - 1))] = j;
            }
            at += __popc(taken[q]);
        }
    }
}

// For every edge (a, b) removed in round r, every triangle {a, b, w} still
// alive at the start of the round is destroyed: each of its edges that
// survives the round loses one support. A triangle with several edges removed
// in this round is handled once, by the removed edge with the smallest id.
// With `next`, an edge whose support falls from `threshold` to below it is
// listed there: supports only fall by one at a time, so every surviving edge
// that the next round removes is listed exactly once, and that round needs no
// scan of the alive edges.
//
// The shorter of the two lists is walked (the longer one binary-searched) in
// chunks of kPeelChunk entries, one warp per chunk, so that a round that
// removes a few hub edges spreads their lists over the whole GPU instead of
// waiting on one warp per edge.
constexpr uint32_t kPeelChunk = 256;

struct PeelEdge {
    uint32_t a, b;       // the removed edge
    uint32_t x, y;       // the walked end and the searched end
    uint32_t xs, xe, ys, ye;
};

// The graph's CSR (eid == nullptr), or its alive entries after a compaction with
// the u < v entry of each one's edge.
struct LiveCsr {
    const uint32_t* offsets;
    const uint32_t* targets;
    const uint32_t* eid;
};

__device__ __forceinline__ PeelEdge peel_edge(const uint32_t* __restrict__ offsets,
                                              const uint32_t* __restrict__ targets,
                                              const uint32_t* __restrict__ src, uint32_t e) {
    PeelEdge p;
    p.a = src[e];
    p.b = targets[e];
    p.xs = offsets[p.a];
    p.xe = offsets[p.a + 1];
    p.ys = offsets[p.b];
    p.ye = offsets[p.b + 1];
    p.x = p.a;
    p.y = p.b;
    if (p.xe - p.xs > p.ye - p.ys) {
        uint32_t t = p.xs; p.xs = p.ys; p.ys = t;
        t = p.xe; p.xe = p.ye; p.ye = t;
        p.x = p.b;
        p.y = p.a;
    }
    return p;
}

// chunks[i] = the walk chunks of removed edge i: none where its support, the
// triangles alive at the round's start, is 0.
__global__ void kt_peel_chunks_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets,
                                      const uint32_t* __restrict__ src, const uint32_t* __restrict__ support,
                                      const uint32_t* __restrict__ removed,
                                      const uint32_t* __restrict__ removed_count, uint32_t* __restrict__ chunks) {
    const uint32_t n = *removed_count;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t e = removed[i];
        const PeelEdge p = peel_edge(offsets, targets, src, e);
        chunks[i] = support[e] ? (p.xe - p.xs + kPeelChunk - 1) / kPeelChunk : 0u;
    }
}

// Warp per chunk: chunk_start (n + 1 words) is the exclusive scan of the
// chunk counts; each warp finds its edge by a binary search of it.
__global__ void __launch_bounds__(256) kt_peel_kernel(const uint32_t* __restrict__ offsets,
                                                      const uint32_t* __restrict__ targets,
                                                      const uint32_t* __restrict__ src,
                                                      const uint32_t* __restrict__ rev,
                                                      const uint32_t* __restrict__ state,
                                                      uint32_t* __restrict__ support,
                                                      const uint32_t* __restrict__ removed,
                                                      const uint32_t* __restrict__ removed_count,
                                                      const uint32_t* __restrict__ chunk_start, uint32_t round,
                                                      uint32_t threshold, uint32_t* __restrict__ next,
                                                      uint32_t* __restrict__ next_count) {
    const unsigned lane = lane_id();
    const uint32_t n = *removed_count;
    const uint32_t total = chunk_start[n];
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t w = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < total; w += nwarps) {
        // i = the largest index with chunk_start[i] <= w (past edges without chunks).
        uint32_t lo = 0, hi = n;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (chunk_start[mid] <= w)
                lo = mid;
            else
                hi = mid;
        }
        const uint32_t e = removed[lo];
        const PeelEdge pe = peel_edge(offsets, targets, src, e);
        const uint32_t chunk = static_cast<uint32_t>(w) - chunk_start[lo];
        const uint32_t begin = range_begin(pe.xs, kPeelChunk, chunk);
        const uint32_t count = range_end(pe.xs, pe.xe - pe.xs, kPeelChunk, chunk) - begin;
        for (uint32_t o = lane; o < count; o += 32) {
            const uint32_t p = begin + o;
            const uint32_t wv = targets[p];
            if (wv == pe.a || wv == pe.b) continue;
            const uint32_t e1 = pe.x < wv ? p : rev[p];
            const uint32_t s1 = state[e1];
            if (s1 != 0 && s1 != round) continue;
            const uint32_t q = lower_bound_u32(targets, pe.ys, pe.ye, wv);
            if (q == pe.ye || targets[q] != wv) continue;
            const uint32_t e2 = pe.y < wv ? q : rev[q];
            const uint32_t s2 = state[e2];
            if (s2 != 0 && s2 != round) continue;
            if ((s1 == round && e1 < e) || (s2 == round && e2 < e)) continue;
            if (s1 == 0 && atomicSub(support + e1, 1u) == threshold && next) next[atomicAdd(next_count, 1u)] = e1;
            if (s2 == 0 && atomicSub(support + e2, 1u) == threshold && next) next[atomicAdd(next_count, 1u)] = e2;
        }
    }
}

// One peel: chunk counts of the n removed edges, their scan, the chunk walk.
// chunks holds n + 1 words.
static Error launch_peel(DeviceImpl& dev, GraphImpl& g, const uint32_t* src,
                         const uint32_t* rev, const uint32_t* state, uint32_t* support, const uint32_t* list,
                         const uint32_t* count, uint32_t n, uint32_t* chunks, uint32_t round, uint32_t threshold,
                         uint32_t* next, uint32_t* next_count) {
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    const unsigned grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(n, 256), cap)));
    GCU_LAUNCH(dev, "kt_peel_chunks", kt_peel_chunks_kernel, grid, 256, 0, g.offsets.ptr, g.targets.ptr, src, support,
               list, count, chunks);
    GCU_TRY(exclusive_scan_u32(dev, chunks, chunks, n));
    GCU_LAUNCH(dev, "kt_peel", kt_peel_kernel, static_cast<unsigned>(cap), 256, 0, g.offsets.ptr, g.targets.ptr, src, rev,
               state, support, list, count, chunks, round, threshold, next, next_count);
    return ok();
}

// ---------------------------------------------------------------- live CSR compaction

// keep[p] for every live entry p = u -> w: not a self-loop and its edge alive
// (state 0, or `pending`: removed in the next round only).
__global__ void __launch_bounds__(256) kt_live_flag_kernel(const LiveCsr lv, uint32_t V, uint32_t L,
                                                           const uint32_t* __restrict__ rev,
                                                           const uint32_t* __restrict__ state, uint32_t pending,
                                                           uint32_t* __restrict__ keep) {
    for_each_entry<256, 4>(lv.offsets, V, L, [&](uint32_t p, uint32_t u) {
        const uint32_t w = lv.targets[p];
        const uint32_t s = u != w ? state[lv.eid ? lv.eid[p] : u < w ? p : rev[p]] : 1u;
        keep[p] = (u != w && (s == 0 || (pending && s == pending))) ? 1u : 0u;
    });
}

__global__ void kt_live_offsets_kernel(const uint32_t* __restrict__ offsets, uint32_t V,
                                       const uint32_t* __restrict__ pos, uint32_t* __restrict__ out) {
    for (uint64_t u = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; u <= V;
         u += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        out[u] = pos[offsets[u]];
}

// eid: the u < v entry, in the graph's CSR, of the edge of each live entry.
__global__ void __launch_bounds__(256) kt_live_fill_kernel(const LiveCsr lv, uint32_t V, uint32_t L,
                                                           const uint32_t* __restrict__ rev,
                                                           const uint32_t* __restrict__ pos,
                                                           uint32_t* __restrict__ targets,
                                                           uint32_t* __restrict__ eid) {
    for_each_entry<256, 4>(lv.offsets, V, L, [&](uint32_t p, uint32_t u) {
        const uint32_t at = pos[p];
        if (pos[p + 1] == at) return;
        const uint32_t w = lv.targets[p];
        targets[at] = w;
        eid[at] = lv.eid ? lv.eid[p] : u < w ? p : rev[p];
    });
}

// The alive entries of `lv` (L entries) in a new CSR (same order), so that
// the peel of later rounds walks alive lists only.
struct LiveBuffers {
    DeviceBuffer<uint32_t> offsets, targets, eid;
    uint32_t entries = 0;
    // Dense form (live_matrix): the vertices with entries numbered in order, and
    // a row of neighbour bits for each.
    DeviceBuffer<uint32_t> number;   // of every vertex
    DeviceBuffer<uint32_t> bits;     // n_rows x words
    DeviceBuffer<uint16_t> before;   // bits of the row in the words before
    DeviceBuffer<ushort2> span;      // the row's words [x, y) hold all its bits
    DeviceBuffer<uint16_t> numbers;  // of the live entries' vertices
    uint32_t words = 0;              // 0: not built
};

// entries: the alive ones, two per alive edge. Known, so nothing waits for a count: for
// graphs without triangles that wait was a fifth of the decomposition (4,096 vertices
// of a grid 126 -> 95 us, with its buffers in two allocations).
static Error compact_live(DeviceImpl& dev, uint32_t V, const LiveCsr& lv, uint32_t L, const uint32_t* rev,
                          const uint32_t* state, uint32_t entries, LiveBuffers* out, uint32_t pending = 0) {
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    DeviceBuffer<uint32_t> pos;
    GCU_TRY(pos.allocate(dev, static_cast<uint64_t>(L) + 1));
    GCU_TRY(out->offsets.allocate(dev, static_cast<uint64_t>(V) + 1));
    const unsigned tiles = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(L, 1024), cap)));
    const unsigned vgrid =
        static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(static_cast<uint64_t>(V) + 1, 256), cap));
    if (L > 0)
        GCU_LAUNCH(dev, "kt_live_flag", kt_live_flag_kernel, tiles, 256, 0, lv, V, L, rev, state, pending, pos.ptr);
    GCU_TRY(exclusive_scan_u32(dev, pos.ptr, pos.ptr, L));
    GCU_LAUNCH(dev, "kt_live_offsets", kt_live_offsets_kernel, vgrid, 256, 0, lv.offsets, V, pos.ptr,
               out->offsets.ptr);
    out->entries = entries;
    GCU_TRY(out->targets.allocate(dev, std::max<uint32_t>(out->entries, 1)));
    GCU_TRY(out->eid.allocate(dev, std::max<uint32_t>(out->entries, 1)));
    if (out->entries > 0)
        GCU_LAUNCH(dev, "kt_live_fill", kt_live_fill_kernel, tiles, 256, 0, lv, V, L, rev, pos.ptr, out->targets.ptr,
                   out->eid.ptr);
    return ok();  // pos is freed in stream order
}

// Number and row bit of every live entry.
__global__ void __launch_bounds__(256) kt_matrix_bits_kernel(const uint32_t* __restrict__ offsets,
                                                             const uint32_t* __restrict__ targets, uint32_t V,
                                                             uint32_t L, const uint32_t* __restrict__ number,
                                                             uint32_t words, uint16_t* __restrict__ numbers,
                                                             uint32_t* __restrict__ bits) {
    for_each_entry<256, 4>(offsets, V, L, [&](uint32_t p, uint32_t u) {
        const uint32_t w = number[targets[p]];
        numbers[p] = static_cast<uint16_t>(w);
        atomicOr(bits + static_cast<uint64_t>(number[u]) * words + (w >> 5), 1u << (w & 31));
    });
}

// A warp per row: the bits before each word, and the words between its first
// and last bits.
__global__ void __launch_bounds__(256) kt_matrix_before_kernel(const uint32_t* __restrict__ bits, uint32_t rows,
                                                               uint32_t words, uint16_t* __restrict__ before,
                                                               ushort2* __restrict__ span) {
    const unsigned lane = lane_id();
    for (uint64_t r = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < rows;
         r += (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5) {
        uint32_t total = 0, first = words, last = 0;
        for (uint32_t j0 = 0; j0 < words; j0 += 32) {
            const uint32_t j = j0 + lane;
            const uint32_t n = j < words ? __popc(bits[r * words + j]) : 0u;
            const uint32_t upto = warp_inclusive_scan(n);
            if (j < words) before[r * words + j] = static_cast<uint16_t>(total + upto - n);
            if (n) {
                first = min(first, j);
                last = j + 1;
            }
            total += __shfl_sync(kFullMask, upto, 31);
        }
        first = __reduce_min_sync(kFullMask, first);
        last = __reduce_max_sync(kFullMask, last);
        if (lane == 0) span[r] = make_ushort2(static_cast<uint16_t>(first), static_cast<uint16_t>(last));
    }
}

__global__ void kt_has_entries_kernel(const uint32_t* __restrict__ offsets, uint32_t V, uint32_t* __restrict__ has) {
    for (uint64_t u = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; u < V;
         u += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        has[u] = offsets[u + 1] > offsets[u] ? 1u : 0u;
}

// The dense form of the live lists, where intersecting two rows' words is less
// work than searching: W words of two rows are 2 W / 32 coalesced loads of a
// warp, d entries searched in a list of their kind d / 32 walks of 10 or more
// dependent, scattered ones. Left out (words = 0) for more vertices than 16-bit
// positions allow, for rows of more than kDenseWords words per live neighbour,
// and where there is no memory for it.
constexpr uint32_t kDenseRows = 65535;
constexpr uint32_t kDenseWords = 8;
constexpr uint32_t kDenseEntries = 65536;  // live entries that are worth its launches

static Error live_matrix(DeviceImpl& dev, uint32_t V, LiveBuffers* lv) {
    lv->words = 0;
    if (lv->entries < kDenseEntries) return ok();
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    GCU_TRY(lv->number.allocate(dev, static_cast<uint64_t>(V) + 1));
    GCU_LAUNCH(dev, "kt_has_entries", kt_has_entries_kernel,
               static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(V, 256), cap)), 256, 0, lv->offsets.ptr, V,
               lv->number.ptr);
    GCU_TRY(exclusive_scan_u32(dev, lv->number.ptr, lv->number.ptr, V));
    uint32_t rows = 0;
    GCU_CUDA(cudaMemcpyAsync(&rows, lv->number.ptr + V, sizeof(uint32_t), cudaMemcpyDeviceToHost, dev.stream), "copy");
    GCU_TRY(dev.sync());
    const uint32_t words = static_cast<uint32_t>(ceil_div_u64(rows, 32));
    if (rows > kDenseRows || static_cast<uint64_t>(words) * rows > static_cast<uint64_t>(kDenseWords) * lv->entries)
        return ok();
    const uint64_t all = static_cast<uint64_t>(rows) * words;
    if (!lv->bits.allocate(dev, all).ok() || !lv->before.allocate(dev, all).ok() ||
        !lv->span.allocate(dev, rows).ok() || !lv->numbers.allocate(dev, lv->entries).ok()) {
        lv->bits.reset();
        lv->before.reset();
        return ok();
    }
    GCU_CUDA(cudaMemsetAsync(lv->bits.ptr, 0, sizeof(uint32_t) * all, dev.stream), "memset");
    GCU_LAUNCH(dev, "kt_matrix_bits", kt_matrix_bits_kernel,
               static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(lv->entries, 1024), cap)), 256, 0,
               lv->offsets.ptr, lv->targets.ptr, V, lv->entries, lv->number.ptr, words,
               lv->numbers.ptr, lv->bits.ptr);
    GCU_LAUNCH(dev, "kt_matrix_before", kt_matrix_before_kernel,
               static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(rows, 8), cap)), 256, 0, lv->bits.ptr, rows,
               words, lv->before.ptr, lv->span.ptr);
    lv->words = words;
    return ok();
}

// The entries listed for round r are removed in it (state = r).
__global__ void kt_mark_kernel(const uint32_t* __restrict__ list, const uint32_t* __restrict__ count,
                               uint32_t* __restrict__ state, uint32_t round) {
    const uint32_t n = *count;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        state[list[i]] = round;
}

// Compacts the alive u < v entries, in CSR order, into host pairs.
template <class Alive>
static Error emit_edges(DeviceImpl& dev, GraphImpl& g, const uint32_t* src, Alive alive, uint32_t* flag,
                        uint32_t* pos, HostArray* edges) {
    const uint32_t E = g.num_edges;
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    const unsigned edge_grid = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(E, 256), cap));
    GCU_LAUNCH(dev, "kt_flag", kt_flag_kernel<Alive>, edge_grid, 256, 0, g.targets.ptr, src, alive, E, flag);
    GCU_TRY(exclusive_scan_u32(dev, flag, pos, E));
    uint32_t count = 0;
    GCU_CUDA(cudaMemcpyAsync(&count, pos + E, sizeof(uint32_t), cudaMemcpyDeviceToHost, dev.stream), "copy");
    GCU_TRY(dev.sync());
    if (count > 0) {
        DeviceBuffer<uint2> out;
        GCU_TRY(out.allocate(dev, count));
        GCU_LAUNCH(dev, "kt_emit", kt_emit_kernel<Alive>, edge_grid, 256, 0, g.targets.ptr, src, alive, E, pos,
                   out.ptr);
        GCU_TRY(edges->resize(2 * static_cast<size_t>(count)));
        GCU_TRY(copy_to_host(dev, edges->data(), out.ptr, sizeof(uint2) * count));
    }
    return ok();
}

// Any CSR: the reference's rounds, recomputing every support each round.
static Error k_truss_general(GraphImpl& g, uint32_t k, const uint32_t* src, const uint32_t* rev,
                             HostArray* edges, uint32_t* iterations) {
    DeviceImpl& dev = *g.dev;
    const uint32_t E = g.num_edges;
    const uint32_t threshold = k - 2;
    DeviceBuffer<uint32_t> support, pos, scratch;
    DeviceBuffer<uint8_t> live;
    GCU_TRY(support.allocate(dev, E));
    GCU_TRY(pos.allocate(dev, static_cast<uint64_t>(E) + 1));
    GCU_TRY(live.allocate(dev, E));
    GCU_TRY(scratch.allocate(dev, 1));
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    const unsigned edge_grid = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(E, 256), cap));
    GCU_CUDA(cudaMemsetAsync(live.ptr, 1, E, dev.stream), "memset");
    uint32_t rounds = 0;
    while (true) {
        GCU_CUDA(cudaMemsetAsync(support.ptr, 0, sizeof(uint32_t) * static_cast<size_t>(E), dev.stream), "memset");
        GCU_LAUNCH(dev, "kt_support", kt_support_kernel, edge_grid, 256, 0, g.offsets.ptr, g.targets.ptr, src, rev,
                   live.ptr, E, support.ptr);
        GCU_CUDA(cudaMemsetAsync(scratch.ptr, 0, sizeof(uint32_t), dev.stream), "memset");
        GCU_LAUNCH(dev, "kt_filter", kt_filter_kernel, edge_grid, 256, 0, support.ptr, live.ptr, E, threshold,
                   scratch.ptr);
        uint32_t removed = 0;
        GCU_CUDA(cudaMemcpyAsync(&removed, scratch.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, dev.stream), "copy");
        GCU_TRY(dev.sync());
        rounds += 1;
        if (removed == 0) break;
    }
    *iterations = rounds;
    return emit_edges(dev, g, src, LiveFlag{live.ptr}, support.ptr, pos.ptr, edges);
}

// Per-graph state of the symmetric k-truss: row of every entry, reverse
// entries, self-loop flags and the triangle support of every u < v entry. It
// depends only on the graph, so it is computed once and reused by every
// k_truss call and by the truss decomposition (3 E + V words of HBM, kept
// with the graph like the PageRank plan).
struct KtCache {
    DeviceBuffer<uint32_t> src, rev, support;
    DeviceBuffer<uint8_t> loop;
    uint32_t loops = 0;  // self-loop entries
};

void destroy_kt_cache(KtCache* c) { delete c; }

static Error ensure_kt_cache(GraphImpl& g, KtCache** out) {
    if (!g.kt_cache) {
        DeviceImpl& dev = *g.dev;
        const uint32_t E = g.num_edges, V = g.num_nodes;
        auto c = std::unique_ptr<KtCache, void (*)(KtCache*)>(new KtCache, destroy_kt_cache);
        GCU_TRY(c->src.allocate(dev, E));
        GCU_TRY(c->rev.allocate(dev, E));
        GCU_TRY(c->support.allocate(dev, E));
        GCU_TRY(c->loop.allocate(dev, V));
        DeviceBuffer<uint32_t> count;
        GCU_TRY(count.allocate(dev, 1));
        const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
        const unsigned tile_grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(E, 1024), cap)));
        const unsigned edge_grid = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(E, 256), cap));
        GCU_LAUNCH(dev, "kt_rows", kt_rows_kernel, tile_grid, 256, 0, g.offsets.ptr, V, E, c->src.ptr);
        GCU_LAUNCH(dev, "kt_pairs", kt_pairs_kernel, edge_grid, 256, 0, g.offsets.ptr, g.targets.ptr, c->src.ptr, E,
                   c->rev.ptr);
        GCU_CUDA(cudaMemsetAsync(c->loop.ptr, 0, V, dev.stream), "memset");
        GCU_CUDA(cudaMemsetAsync(count.ptr, 0, sizeof(uint32_t), dev.stream), "memset");
        GCU_LAUNCH(dev, "kt_loops", kt_loops_kernel, edge_grid, 256, 0, g.targets.ptr, c->src.ptr, E, c->loop.ptr,
                   count.ptr);
        GCU_CUDA(cudaMemsetAsync(c->support.ptr, 0, sizeof(uint32_t) * static_cast<size_t>(E), dev.stream), "memset");
        GCU_TRY(edge_support(g, c->rev.ptr, c->support.ptr));
        GCU_CUDA(cudaMemcpyAsync(&c->loops, count.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, dev.stream), "copy");
        GCU_TRY(dev.sync());
        g.kt_cache = c.release();
    }
    *out = g.kt_cache;
    return ok();
}

// Symmetric CSR: per-edge triangle counts (cached), then
// incremental peeling. Every round removes exactly the entries the
// reference's round removes, so the edge list and the round count are the
// same.
static Error k_truss_symmetric(GraphImpl& g, uint32_t k, HostArray* edges, uint32_t* iterations) {
    DeviceImpl& dev = *g.dev;
    const uint32_t E = g.num_edges;
    const uint32_t threshold = k - 2;
    KtCache* c = nullptr;
    GCU_TRY(ensure_kt_cache(g, &c));
    const uint32_t* src = c->src.ptr;
    const uint32_t* rev = c->rev.ptr;
    DeviceBuffer<uint32_t> support, state, removed, scratch, lists[2];
    GCU_TRY(support.allocate(dev, static_cast<uint64_t>(E) + 1));
    GCU_TRY(state.allocate(dev, static_cast<uint64_t>(E) + 1));
    GCU_TRY(removed.allocate(dev, E));
    GCU_TRY(lists[0].allocate(dev, E));
    GCU_TRY(lists[1].allocate(dev, E));
    DeviceBuffer<uint32_t> chunks;  // peel chunk counts, then their scan
    GCU_TRY(chunks.allocate(dev, static_cast<uint64_t>(E) + 1));
    GCU_TRY(scratch.allocate(dev, 3));  // [0] removed by a scan, [1 + b] entries of lists[b]
    GCU_CUDA(cudaMemcpyAsync(support.ptr, c->support.ptr, sizeof(uint32_t) * static_cast<size_t>(E),
                             cudaMemcpyDeviceToDevice, dev.stream),
             "copy");
    GCU_CUDA(cudaMemsetAsync(state.ptr, 0, sizeof(uint32_t) * static_cast<size_t>(E), dev.stream), "memset");
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    const unsigned edge_grid = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(E, 256), cap));
    const uint32_t loops = c->loops;

    // Rounds 1 and (with self-loops) 2 scan every entry: round 1 adds the
    // self-loop terms, so an edge it keeps may be below the threshold in
    // round 2 without losing a triangle. Later rounds remove exactly the
    // edges that the previous round's peel brought below the threshold.
    uint32_t round = 1;
    int cur = 0;       // the peel of this round lists the next round's removals in lists[cur]
    uint32_t n = 0;    // entries removed in this round
    while (true) {
        const bool scan = round == 1 || (round == 2 && loops > 0);
        const uint32_t* list = removed.ptr;
        const uint32_t* count = scratch.ptr;
        if (scan) {
            GCU_CUDA(cudaMemsetAsync(scratch.ptr, 0, sizeof(uint32_t), dev.stream), "memset");
            GCU_LAUNCH(dev, "kt_round_filter", kt_round_filter_kernel, edge_grid, 256, 0, g.targets.ptr, src,
                       c->loop.ptr, support.ptr, state.ptr, E, threshold, round, removed.ptr, scratch.ptr);
            GCU_CUDA(cudaMemcpyAsync(&n, scratch.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, dev.stream), "copy");
            GCU_TRY(dev.sync());
        } else {
            // n = the previous peel's list (read below); mark it removed in this round.
            list = lists[cur ^ 1].ptr;
            count = scratch.ptr + 1 + (cur ^ 1);
            if (n > 0) {
                const unsigned grid =
                    static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(n, 256), cap));
                GCU_LAUNCH(dev, "kt_mark", kt_mark_kernel, grid, 256, 0, list, count, state.ptr, round);
            }
        }
        // Round 1 also removes the self-loop entries (their support is 0).
        const bool removed_any = n > 0 || (round == 1 && loops > 0);
        if (!removed_any) break;
        uint32_t next_n = 0;
        GCU_CUDA(cudaMemsetAsync(scratch.ptr + 1 + cur, 0, sizeof(uint32_t), dev.stream), "memset");
        if (n > 0) {
            GCU_TRY(launch_peel(dev, g, src, rev, state.ptr, support.ptr, list, count, n, chunks.ptr, round, threshold, lists[cur].ptr,
                                scratch.ptr + 1 + cur));
            GCU_CUDA(cudaMemcpyAsync(&next_n, scratch.ptr + 1 + cur, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                     dev.stream),
                     "copy");
            GCU_TRY(dev.sync());
        }
        n = next_n;
        cur ^= 1;
        round += 1;
    }
    *iterations = round;
    // `removed` (E entries) and `support` (E + 1) are reused as the compaction's flag and scan buffers.
    return emit_edges(dev, g, src, RoundState{state.ptr}, removed.ptr, support.ptr, edges);
}

Error k_truss(GraphImpl& g, uint32_t k, HostArray* edges, uint32_t* iterations) {
    GCU_TRY(edges->resize(0));
    *iterations = 0;
    const uint32_t E = g.num_edges, V = g.num_nodes;
    // k_truss.rs:53-60: no edges, no truss.
    if (E == 0) return ok();
    DeviceImpl& dev = *g.dev;
    bool symmetric = false;
    GCU_TRY(graph_symmetry(g, &symmetric));
    if (symmetric) return k_truss_symmetric(g, k, edges, iterations);
    DeviceBuffer<uint32_t> src, rev;
    GCU_TRY(src.allocate(dev, E));
    GCU_TRY(rev.allocate(dev, E));
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    const unsigned tile_grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(E, 1024), cap)));
    const unsigned edge_grid = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(E, 256), cap));
    GCU_LAUNCH(dev, "kt_rows", kt_rows_kernel, tile_grid, 256, 0, g.offsets.ptr, V, E, src.ptr);
    GCU_LAUNCH(dev, "kt_reverse", kt_reverse_kernel, edge_grid, 256, 0, g.offsets.ptr, g.targets.ptr, src.ptr, E,
               rev.ptr);
    return k_truss_general(g, k, src.ptr, rev.ptr, edges, iterations);
}

// ---------------------------------------------------------------- truss decomposition

// Appends, warp-aggregated, the entries with take set (all 32 lanes call it).
__device__ __forceinline__ void kt_append(bool take, uint32_t j, uint32_t* __restrict__ list,
                                          uint32_t* __restrict__ count) {
    const unsigned mask = __ballot_sync(kFullMask, take);
    if (mask == 0) return;
    const unsigned lane = lane_id();
    const int leader = __ffs(mask) - 1;
    uint32_t at = 0;
    if (lane == static_cast<unsigned>(leader)) at = atomicAdd(count, static_cast<uint32_t>(__popc(mask)));
    at = __shfl_sync(kFullMask, at, leader);
    if (take) list[at + __popc(mask & ((1u << lane) - 1))] = j;
}

// The alive u < v entries: from all E entries (list == nullptr) or from a
// previous active list of n entries.
__global__ void kt_active_kernel(const uint32_t* __restrict__ targets, const uint32_t* __restrict__ src,
                                 const uint32_t* __restrict__ state, const uint32_t* __restrict__ list, uint32_t n,
                                 uint32_t* __restrict__ out, uint32_t* __restrict__ count) {
    for (uint64_t base = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) & ~31ull; base < n;
         base += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t i = base + lane_id();
        bool take = false;
        uint32_t j = 0;
        if (i < n) {
            j = list ? list[i] : static_cast<uint32_t>(i);
            take = state[j] == 0 && targets[j] > src[j];
        }
        kt_append(take, j, out, count);
    }
}

// The decomposition's rounds run in one cooperative launch, from one compaction
// of the live lists to the next; the blocks meet at a grid barrier after every
// scan and every peel. State of an edge (its u < v entry): 0 alive, r removed in
// round r; the peel of round r marks what round r + 1 removes with r + 1 when it
// lists it, so during round r an edge is alive if its state is 0 or r + 1.
struct TrussState {
    GridBarrier bar;
    uint32_t count[3];  // entries listed by the phase, rotating (slot p % 3 is phase p's)
    uint32_t least[3];  // smallest support a scan left alive
    uint32_t longs[3];  // edges put off by the phase
    // carried from launch to launch
    uint32_t k, round, top, phase, level_start, list, n;
    uint32_t alive;
};

struct TrussLoop {
    const uint32_t* offsets;  // live CSR
    const uint32_t* targets;
    const uint32_t* eid;      // u < v entry (in the graph's CSR) of each live entry
    const uint32_t* number;   // the dense form (words > 0)
    const uint32_t* bits;
    const uint16_t* before;
    const ushort2* span;
    const uint16_t* numbers;
    uint32_t words;
    const uint32_t* g_targets;
    const uint32_t* src;
    uint32_t* state;
    uint32_t* support;
    uint32_t* truss;
    const uint32_t* active;
    uint32_t listed;
    uint32_t* list0;
    uint32_t* list1;
    uint32_t* longs;          // edges put off
    TrussState* st;
};

// What bounds the loop: R-MAT scale 19 (14.3 M entries, trussness up to 187,
// 1,697 rounds) takes 132 scans and about 1,300 peels. A round of a few edges is
// one peel's chain of dependent loads and the barrier, 4 to 8 us; in larger rounds
// it is the triangles' scattered loads and atomics, and before the dense form
// (first 108 rounds) the searches. Measured there, the whole decomposition after
// the support: 109.5 ms when each round was four launches and a count read by the
// host, 40.7 in this loop with searched lists only (nine in ten were too long for
// the stage), 35.1 with rows intersected, 28.7 with short lists looked up in rows,
// 28.0 with a scan's four edges per lane taken with one atomic. With 1, 2, 3 or 8
// words intersected per walked entry saved 28.6, 28.7, 28.7, 31.5 ms.
constexpr int kTrussThreads = 1024;
constexpr uint32_t kStage = 512;  // entries of the searched list a warp stages in shared memory
constexpr int kTrussUnroll = 2;   // walked entries per lane in flight
constexpr int kScanLoads = 4;     // listed edges per lane in flight in a scan
// An edge of which a warp would walk more than this many entries is put off, and
// the round's edges of that kind are then shared by all warps. Else a hub's edge is
// one warp's while the others wait at the barrier: 4 hubs of 600,000 leaves, joined
// to one another, 44.9 -> 11.7 ms. Limits of 2,048, 8,192 and 32,768 entries are alike
// (R-MAT 19 30.6 to 31.9 ms with and without).
constexpr uint32_t kLongWalk = 8192;
// Active edges that are not worth a compaction (some 100 us of launches and waits):
// 2,000 vertices and 16,000 edges 0.49 -> 0.17 ms with kDenseEntries, R-MAT 14 5.5 ->
// 4.5; with 32,768 edges 0.17 and 4.7, with 524,288 0.17 and 5.0.
constexpr uint32_t kCompactEdges = 131072;
constexpr uint32_t kMaxLogParts = 12;

// Removes, with edge e, the triangles it makes with the live entries p1 and p2
// (where hit). A triangle with several edges removed in this round is handled
// once, by the one with the smallest id; the edges of it that survive the round
// lose one support, and one that falls below the threshold is listed for the
// next round.
__device__ __forceinline__ void truss_remove(const TrussLoop& a, uint32_t e, const bool (&hit)[kTrussUnroll],
                                             const uint32_t (&p1)[kTrussUnroll], const uint32_t (&p2)[kTrussUnroll],
                                             uint32_t round, uint32_t k, uint32_t* next, uint32_t* next_count) {
    uint32_t e1[kTrussUnroll], e2[kTrussUnroll], s1[kTrussUnroll], s2[kTrussUnroll];
#pragma unroll
    for (int c = 0; c < kTrussUnroll; ++c) {
        e1[c] = ld_nc_if(hit[c], a.eid + p1[c], 0u);
        e2[c] = ld_nc_if(hit[c], a.eid + p2[c], 0u);
    }
#pragma unroll
    for (int c = 0; c < kTrussUnroll; ++c) {
        s1[c] = ld_if(hit[c], a.state + e1[c], 1u);
        s2[c] = ld_if(hit[c], a.state + e2[c], 1u);
    }
#pragma unroll
    for (int c = 0; c < kTrussUnroll; ++c) {
        if (!hit[c]) continue;
        const bool live1 = s1[c] == 0 || s1[c] == round + 1, live2 = s2[c] == 0 || s2[c] == round + 1;
        if ((!live1 && s1[c] != round) || (!live2 && s2[c] != round)) continue;   // destroyed earlier
        if ((!live1 && e1[c] < e) || (!live2 && e2[c] < e)) continue;             // another edge's triangle
        if (live1 && atomicSub(a.support + e1[c], 1u) == k - 2) {
            a.state[e1[c]] = round + 1;
            a.truss[e1[c]] = k - 1;
            next[atomicAdd(next_count, 1u)] = e1[c];
        }
        if (live2 && atomicSub(a.support + e2[c], 1u) == k - 2) {
            a.state[e2[c]] = round + 1;
            a.truss[e2[c]] = k - 1;
            next[atomicAdd(next_count, 1u)] = e2[c];
        }
    }
}

// One removed edge (or the part-th of 2^log_parts slices of its walk): the
// shorter live list is walked, the longer one searched, in shared memory where
// it fits kStage entries. With `put_off`, a long walk is only listed there.
__device__ __forceinline__ void truss_peel(const TrussLoop& a, uint32_t e, uint32_t part, uint32_t log_parts,
                                           uint32_t round, uint32_t k, uint32_t* s_y, uint32_t* next,
                                           uint32_t* next_count, uint32_t* put_off) {
    const unsigned lane = lane_id();
    const uint32_t u = __ldg(a.src + e), v = __ldg(a.g_targets + e);
    uint32_t xs = __ldg(a.offsets + u), xn = __ldg(a.offsets + u + 1) - xs;
    uint32_t ys = __ldg(a.offsets + v), yn = __ldg(a.offsets + v + 1) - ys;
    if (xn > yn) {
        uint32_t t = xs; xs = ys; ys = t;
        t = xn; xn = yn; yn = t;
    }
    if (put_off && xn >> log_parts > kLongWalk) {
        if (part == 0 && lane == 0) a.longs[atomicAdd(put_off, 1u)] = e;
        return;
    }
    const bool staged = yn <= kStage;
    if (staged) {
        __syncwarp();
#pragma unroll 4
        for (uint32_t i = lane; i < yn; i += 32) s_y[i] = __ldg(a.targets + ys + i);
        __syncwarp();
    }
    const uint32_t steps = yn ? 32 - __clz(yn) : 0;
    const uint32_t stride = 32u << log_parts;
    for (uint32_t i0 = part * 32 + lane; i0 < xn; i0 += kTrussUnroll * stride) {
        uint32_t w[kTrussUnroll], q[kTrussUnroll];
        bool hit[kTrussUnroll];
#pragma unroll
        for (int c = 0; c < kTrussUnroll; ++c) {
            hit[c] = xn - i0 > c * stride;
            w[c] = hit[c] ? __ldg(a.targets + xs + i0 + c * stride) : 0u;
            q[c] = 0;
        }
        // q = entries of the list below w: the list's first entry >= w.
        for (uint32_t b = steps; b-- > 0;) {
#pragma unroll
            for (int c = 0; c < kTrussUnroll; ++c) {
                const uint32_t m = q[c] + (1u << b);
                if (hit[c] && m <= yn && (staged ? s_y[m - 1] : __ldg(a.targets + ys + m - 1)) < w[c]) q[c] = m;
            }
        }
#pragma unroll
        for (int c = 0; c < kTrussUnroll; ++c)
            hit[c] = hit[c] && q[c] < yn && (staged ? s_y[q[c]] : __ldg(a.targets + ys + q[c])) == w[c];
#pragma unroll
        for (int c = 0; c < kTrussUnroll; ++c) {
            w[c] = xs + i0 + c * stride;
            q[c] += ys;
        }
        truss_remove(a, e, hit, w, q, round, k, next, next_count);
    }
}

// The same on the dense form. Where the words that both rows have bits in are
// few, they are intersected; else the shorter live list is walked and each of its
// vertices looked up in the other end's row, one load where a search takes ten or
// more. kDenseLoads words or entries per lane are in flight, and the common
// neighbours' positions in the two live lists are queued in shared memory, from
// where all lanes take them.
constexpr int kDenseLoads = 4;
constexpr uint32_t kWalkWords = 2;  // words intersected per walked entry saved
constexpr uint32_t kDenseBatch = 32 * kTrussUnroll;
constexpr uint32_t kQueue = 32 * 32 + kDenseBatch;  // positions a warp queues: a word per lane beyond a batch

__device__ __forceinline__ void truss_peel_dense(const TrussLoop& a, uint32_t e, uint32_t part, uint32_t log_parts,
                                                 uint32_t round, uint32_t k, uint32_t* s_queue, uint32_t* next,
                                                 uint32_t* next_count, uint32_t*) {
    const unsigned lane = lane_id();
    uint32_t u = __ldg(a.src + e), v = __ldg(a.g_targets + e);
    uint32_t pu = __ldg(a.offsets + u), du = __ldg(a.offsets + u + 1) - pu;
    uint32_t pv = __ldg(a.offsets + v), dv = __ldg(a.offsets + v + 1) - pv;
    uint32_t nu = __ldg(a.number + u), nv = __ldg(a.number + v);
    if (du > dv) {  // u: the shorter list
        uint32_t t = pu; pu = pv; pv = t;
        t = du; du = dv; dv = t;
        t = nu; nu = nv; nv = t;
    }
    const ushort2 su = __ldg(a.span + nu), sv = __ldg(a.span + nv);
    const uint64_t rv = static_cast<uint64_t>(nv) * a.words;
    const uint32_t first = max(su.x, sv.x), last = max(first, static_cast<uint32_t>(min(su.y, sv.y)));
    uint32_t queued = 0;
    auto take = [&](uint32_t n) {  // the last n queued, at most kDenseBatch
        queued -= n;
        __syncwarp();
        bool hit[kTrussUnroll];
        uint32_t p1[kTrussUnroll], p2[kTrussUnroll];
#pragma unroll
        for (int c = 0; c < kTrussUnroll; ++c) {
            hit[c] = lane + c * 32 < n;
            const uint32_t x = hit[c] ? s_queue[queued + lane + c * 32] : 0u;
            p1[c] = pu + (x >> 16);
            p2[c] = pv + (x & 0xFFFFu);
        }
        __syncwarp();
        truss_remove(a, e, hit, p1, p2, round, k, next, next_count);
    };
    const bool intersect = last - first <= kWalkWords * du;
    const uint32_t all = intersect ? last - first : du;
    const uint32_t share = (all + (1u << log_parts) - 1) >> log_parts;  // of this part
    const uint32_t begin = min(part * share, all), end = min(begin + share, all);
    if (intersect) {
        const uint64_t ru = static_cast<uint64_t>(nu) * a.words;
        for (uint32_t j0 = begin; j0 < end; j0 += kDenseLoads * 32) {
            uint32_t x[kDenseLoads], y[kDenseLoads], bx[kDenseLoads], by[kDenseLoads];
#pragma unroll
            for (int c = 0; c < kDenseLoads; ++c) {
                const uint32_t j = j0 + c * 32 + lane;
                x[c] = ld_nc_if(j < end, a.bits + ru + first + j, 0u);
                y[c] = ld_nc_if(j < end, a.bits + rv + first + j, 0u);
            }
#pragma unroll
            for (int c = 0; c < kDenseLoads; ++c) {
                const uint32_t j = j0 + c * 32 + lane;
                bx[c] = x[c] & y[c] ? __ldg(a.before + ru + first + j) : 0u;
                by[c] = x[c] & y[c] ? __ldg(a.before + rv + first + j) : 0u;
            }
#pragma unroll
            for (int c = 0; c < kDenseLoads; ++c) {
                uint32_t m = x[c] & y[c];
                if (!__any_sync(kFullMask, m)) continue;
                const uint32_t n = __popc(m);
                const uint32_t upto = warp_inclusive_scan(n);
                uint32_t at = queued + upto - n;
                for (; m; m &= m - 1) {
                    const uint32_t below = (m & (0u - m)) - 1;
                    s_queue[at++] = (bx[c] + __popc(x[c] & below)) << 16 | (by[c] + __popc(y[c] & below));
                }
                queued += __shfl_sync(kFullMask, upto, 31);
                while (queued >= kDenseBatch) take(kDenseBatch);
            }
        }
    } else {
        for (uint32_t i0 = begin; i0 < end; i0 += kDenseLoads * 32) {
            uint32_t w[kDenseLoads], y[kDenseLoads], by[kDenseLoads];
#pragma unroll
            for (int c = 0; c < kDenseLoads; ++c) {
                const uint32_t i = i0 + c * 32 + lane;
                w[c] = i < end ? __ldg(a.numbers + pu + i) : 0u;
            }
#pragma unroll
            for (int c = 0; c < kDenseLoads; ++c)
                y[c] = ld_nc_if(i0 + c * 32 + lane < end, a.bits + rv + (w[c] >> 5), 0u);
#pragma unroll
            for (int c = 0; c < kDenseLoads; ++c)
                by[c] = (y[c] >> (w[c] & 31)) & 1u ? __ldg(a.before + rv + (w[c] >> 5)) : 0u;
#pragma unroll
            for (int c = 0; c < kDenseLoads; ++c) {
                const bool hit = (y[c] >> (w[c] & 31)) & 1u;
                const unsigned hits = __ballot_sync(kFullMask, hit);
                if (hit)
                    s_queue[queued + __popc(hits & ((1u << lane) - 1))] =
                        (i0 + c * 32 + lane) << 16 | (by[c] + __popc(y[c] & ((1u << (w[c] & 31)) - 1)));
                queued += __popc(hits);
                if (queued >= kDenseBatch) take(kDenseBatch);
            }
        }
    }
    if (queued) take(queued);
}

template <bool kDense>
__global__ void __launch_bounds__(kTrussThreads, 1) kt_truss_loop_kernel(const TrussLoop a) {
    extern __shared__ uint32_t s_stage[];
    __shared__ uint32_t s_count, s_least, s_long;
    const unsigned lane = lane_id();
    uint32_t* s_warp = s_stage + (threadIdx.x >> 5) * (kDense ? kQueue : kStage);
    const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t nthreads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint32_t nwarps = static_cast<uint32_t>(nthreads >> 5);
    const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // neighbours on different SMs
    uint32_t k = a.st->k, round = a.st->round, top = a.st->top, phase = a.st->phase, alive = a.st->alive;
    uint32_t list = a.st->list, n = a.st->n;  // the entries this round removes: lists[list][0 .. n)
    bool level_start = a.st->level_start != 0;
    unsigned barriers = 0;
    // Ends a phase: its counts to every block, the slot after next cleared.
    auto end_phase = [&]() -> bool {
        const uint32_t slot = phase % 3;
        const bool ok = grid_barrier(&a.st->bar, gridDim.x, barriers, [&] {
            s_count = __ldcg(a.st->count + slot);
            s_least = __ldcg(a.st->least + slot);
            s_long = __ldcg(a.st->longs + slot);
        });
        ++phase;
        // Slot (phase + 1) % 3 was read two barriers ago.
        if (tid == 0) {
            a.st->count[(phase + 1) % 3] = 0;
            a.st->least[(phase + 1) % 3] = 0xFFFFFFFFu;
            a.st->longs[(phase + 1) % 3] = 0;
        }
        return ok;
    };
    // Half of a long active list gone: the host compacts it and the live lists.
    while (alive > 0 && (a.listed <= kCompactEdges || 2ull * alive >= a.listed)) {
        ++round;
        if (level_start) {
            uint32_t least = 0xFFFFFFFFu;
            for (uint64_t b = tid & ~31ull; b < a.listed; b += kScanLoads * nthreads) {
                uint32_t j[kScanLoads], alive_state[kScanLoads], s[kScanLoads];
#pragma unroll
                for (int c = 0; c < kScanLoads; ++c) {
                    const uint64_t i = b + c * nthreads + lane;
                    j[c] = ld_nc_if(i < a.listed, a.active + i, kNone);
                }
#pragma unroll
                for (int c = 0; c < kScanLoads; ++c) {
                    alive_state[c] = ld_if(j[c] != kNone, a.state + j[c], 1u);
                    s[c] = ld_if(j[c] != kNone, a.support + j[c], 0u);
                }
                unsigned below[kScanLoads];
                uint32_t taken = 0;
#pragma unroll
                for (int c = 0; c < kScanLoads; ++c) {
                    below[c] = __ballot_sync(kFullMask, alive_state[c] == 0 && s[c] < k - 2);
                    taken += __popc(below[c]);
                    if (alive_state[c] == 0 && s[c] >= k - 2) least = min(least, s[c]);
                }
                if (taken == 0) continue;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(a.st->count + phase % 3, taken);
                at = __shfl_sync(kFullMask, at, 0);
#pragma unroll
                for (int c = 0; c < kScanLoads; ++c) {
                    if ((below[c] >> lane) & 1u) {
                        a.state[j[c]] = round;
                        a.truss[j[c]] = k - 1;
                        (list ? a.list1 : a.list0)[at + __popc(below[c] & ((1u << lane) - 1))] = j[c];
                    }
                    at += __popc(below[c]);
                }
            }
            least = __reduce_min_sync(kFullMask, least);
            if (lane == 0 && least != 0xFFFFFFFFu) atomicMin(a.st->least + phase % 3, least);
            if (!end_phase()) return;
            n = s_count;
            if (n == 0) {
                // Every alive edge is in the k-truss, and in those up to k =
                // least + 2: a round each that removes nothing.
                top = s_least + 2;
                round += top - k;
                k = top + 1;
                continue;
            }
        } else if (n == 0) {
            top = k;
            k += 1;
            level_start = true;
            continue;
        }
        alive -= n;
        // With fewer edges than warps, up to 16 warps share one.
        const uint32_t log_parts = n >= nwarps ? 0u : min(4u, 31 - __clz(nwarps / n));
        for (uint64_t w = warp; w < static_cast<uint64_t>(n) << log_parts; w += nwarps) {
            const uint32_t e = __ldcg((list ? a.list1 : a.list0) + (w >> log_parts));
            // An edge's support is its triangles alive at the round's start.
            if (__ldcg(a.support + e) == 0) continue;
            (kDense ? truss_peel_dense : truss_peel)(a, e, static_cast<uint32_t>(w) & ((1u << log_parts) - 1),
                                                     log_parts, round, k, s_warp, list ? a.list0 : a.list1,
                                                     a.st->count + phase % 3, a.st->longs + phase % 3);
        }
        if (!end_phase()) return;
        n = s_count;
        if (!kDense && s_long) {
            // The edges put off, in as many parts as give every warp a few.
            const uint32_t longs = s_long;
            const uint32_t share = 4 * nwarps / longs;
            const uint32_t parts = min(kMaxLogParts, share ? max(4u, 31 - __clz(share)) : 4u);
            for (uint64_t w = warp; w < static_cast<uint64_t>(longs) << parts; w += nwarps)
                truss_peel(a, __ldcg(a.longs + (w >> parts)), static_cast<uint32_t>(w) & ((1u << parts) - 1), parts, round, k,
                           s_warp, (list ? a.list0 : a.list1) + n, a.st->count + phase % 3, nullptr);
            if (!end_phase()) return;
            n += s_count;
        }
        list ^= 1u;
        level_start = false;
    }
    if (tid == 0) {
        a.st->k = k;
        a.st->round = round;
        a.st->top = top;
        a.st->phase = phase;
        a.st->level_start = level_start ? 1u : 0u;
        a.st->list = list;
        a.st->n = n;
        a.st->alive = alive;
    }
}

// Spreads the u < v entries' trussness to every entry: the reverse entry gets
// the same value, self-loops 0.
__global__ void kt_truss_spread_kernel(const uint32_t* __restrict__ targets, const uint32_t* __restrict__ src,
                                       const uint32_t* __restrict__ rev, const uint32_t* __restrict__ truss,
                                       uint32_t E, uint32_t* __restrict__ out) {
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < E;
         j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t u = src[j], v = targets[j];
        out[j] = u == v ? 0u : truss[u < v ? j : rev[j]];
    }
}

template <class Kernel>
static Error fit_truss_loop(Kernel kernel, size_t smem) {
    GCU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
             "cudaFuncSetAttribute");
    int per_sm = 0;
    GCU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTrussThreads, smem), "occupancy");
    if (per_sm < 1) return kernel_error("truss decomposition: the loop kernel does not fit an SM");
    return ok();
}

// Trussness of every edge of a symmetric CSR: the peeling of k_truss_symmetric
// continued level by level without restarting. At level k the rounds remove
// every alive edge with fewer than k - 2 alive triangles until none is left
// below; the edges removed at level k have trussness k - 1. Self-loops take no
// part (they are in no k-truss for k >= 3).
Error truss_decomposition(GraphImpl& g, uint32_t* host_truss, uint32_t* max_truss, uint32_t* rounds) {
    *max_truss = 0;
    *rounds = 0;
    const uint32_t E = g.num_edges;
    if (E == 0) return ok();
    DeviceImpl& dev = *g.dev;
    bool symmetric = false;
    GCU_TRY(graph_symmetry(g, &symmetric));
    if (!symmetric) return kernel_error("truss decomposition needs a symmetric CSR (every u -> v with its v -> u)");
    KtCache* c = nullptr;
    GCU_TRY(ensure_kt_cache(g, &c));
    const uint32_t* src = c->src.ptr;
    const uint32_t* rev = c->rev.ptr;
    DeviceBuffer<uint32_t> support, zeroed, four;
    DeviceBuffer<TrussState> loop_state;
    // Undirected edges: in a symmetric CSR every edge but a self-loop has two
    // entries. The active list holds the alive ones' u < v entries and, with the
    // live lists, is compacted whenever half of it has been peeled, so late
    // rounds only touch the remaining core.
    const uint32_t edges = (E - c->loops) / 2;
    const uint64_t list_cap = std::max<uint32_t>(edges, 1);
    GCU_TRY(support.allocate(dev, E));
    GCU_TRY(zeroed.allocate(dev, 2 * static_cast<uint64_t>(E) + 1));
    GCU_TRY(four.allocate(dev, 4 * list_cap));
    GCU_TRY(loop_state.allocate(dev, 1));
    uint32_t* const state = zeroed.ptr;
    uint32_t* const truss = state + E;
    uint32_t* const count = truss + E;
    uint32_t* const active[2] = {four.ptr, four.ptr + list_cap};
    uint32_t* const lists[2] = {four.ptr + 2 * list_cap, four.ptr + 3 * list_cap};
    const uint64_t cap = static_cast<uint64_t>(dev.sm_count) * 16;
    const unsigned edge_grid = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(E, 256), cap));
    GCU_CUDA(cudaMemcpyAsync(support.ptr, c->support.ptr, sizeof(uint32_t) * static_cast<size_t>(E),
                             cudaMemcpyDeviceToDevice, dev.stream),
             "copy");
    GCU_CUDA(cudaMemsetAsync(zeroed.ptr, 0, sizeof(uint32_t) * zeroed.count, dev.stream), "memset");
    GCU_LAUNCH(dev, "kt_active", kt_active_kernel, edge_grid, 256, 0, g.targets.ptr, src, state,
               static_cast<const uint32_t*>(nullptr), E, active[0], count);
    LiveBuffers live[2];
    GCU_TRY(compact_live(dev, g.num_nodes, LiveCsr{g.offsets.ptr, g.targets.ptr, nullptr}, E, rev, state, 2 * edges,
                         &live[0]));
    GCU_TRY(live_matrix(dev, g.num_nodes, &live[0]));
    constexpr size_t kListSmem = sizeof(uint32_t) * kStage * (kTrussThreads / 32);
    constexpr size_t kDenseSmem = sizeof(uint32_t) * kQueue * (kTrussThreads / 32);
    TrussState st{};
    st.k = 3;
    st.top = edges > 0 ? 2 : 0;
    st.level_start = 1;
    st.alive = edges;
    uint32_t listed = edges;
    int cur = 0;
    while (st.alive > 0) {
        st.bar = GridBarrier{};
        std::fill(st.count, st.count + 3, 0u);
        std::fill(st.least, st.least + 3, 0xFFFFFFFFu);
        std::fill(st.longs, st.longs + 3, 0u);
        st.phase = 0;
        GCU_CUDA(cudaMemcpyAsync(loop_state.ptr, &st, sizeof(st), cudaMemcpyHostToDevice, dev.stream), "copy");
        const LiveBuffers& lv = live[cur];
        const TrussLoop a{lv.offsets.ptr, lv.targets.ptr, lv.eid.ptr,     lv.number.ptr,    lv.bits.ptr,
                          lv.before.ptr,  lv.span.ptr,    lv.numbers.ptr, lv.words,         g.targets.ptr,
                          src,            state,          support.ptr,    truss,            active[cur],
                          listed,         lists[0],       lists[1],       active[cur ^ 1],  loop_state.ptr};
        // One block per SM; fewer for a core too small to use them.
        const unsigned grid = static_cast<unsigned>(std::max<uint64_t>(
            1, std::min<uint64_t>(dev.sm_count, ceil_div_u64(listed, kTrussThreads / 32))));
        if (lv.words) {
            GCU_TRY(fit_truss_loop(kt_truss_loop_kernel<true>, kDenseSmem));
            GCU_LAUNCH_COOP(dev, "kt_truss_dense", kt_truss_loop_kernel<true>, grid, kTrussThreads, kDenseSmem, a);
        } else {
            GCU_TRY(fit_truss_loop(kt_truss_loop_kernel<false>, kListSmem));
            GCU_LAUNCH_COOP(dev, "kt_truss_loop", kt_truss_loop_kernel<false>, grid, kTrussThreads, kListSmem, a);
        }
        GCU_CUDA(cudaMemcpyAsync(&st, loop_state.ptr, sizeof(st), cudaMemcpyDeviceToHost, dev.stream), "copy");
        GCU_TRY(dev.sync());
        if (st.bar.failed) return kernel_error("truss decomposition: a block did not reach the grid barrier");
        if (st.alive == 0) break;
        // The removals listed for the next round count as alive (state round +
        // 1), and their lists stay.
        GCU_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), dev.stream), "memset");
        const unsigned grid_l = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(listed, 256), cap));
        GCU_LAUNCH(dev, "kt_active", kt_active_kernel, grid_l, 256, 0, g.targets.ptr, src, state, active[cur],
                   listed, active[cur ^ 1], count);
        listed = st.alive - st.n;
        GCU_TRY(compact_live(dev, g.num_nodes,
                             LiveCsr{live[cur].offsets.ptr, live[cur].targets.ptr, live[cur].eid.ptr},
                             live[cur].entries, rev, state, 2 * st.alive, &live[cur ^ 1],
                             st.n > 0 ? st.round + 1 : 0));
        GCU_TRY(live_matrix(dev, g.num_nodes, &live[cur ^ 1]));
        cur ^= 1;
    }
    *max_truss = st.top;
    *rounds = st.round;
    if (host_truss) {
        GCU_LAUNCH(dev, "kt_truss_spread", kt_truss_spread_kernel, edge_grid, 256, 0, g.targets.ptr, src, rev,
                   truss, E, support.ptr);
        GCU_TRY(copy_to_host(dev, host_truss, support.ptr, sizeof(uint32_t) * static_cast<size_t>(E)));
    }
    return ok();
}

}  // namespace gcu

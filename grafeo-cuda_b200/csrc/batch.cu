// Batched form: many uneven graphs packed into one CSR and processed by
// persistent kernels, replayed as one captured CUDA graph.
//
// Layout: graph i owns the vertices [vbase[i], vbase[i + 1]) of a union CSR
// whose targets are union ids (no edge leaves its graph), so the union is a
// plain symmetric CSR and graph i's entries are [offsets[vbase[i]],
// offsets[vbase[i + 1]]).
//
//  * Triangles: word lists of the union, counted per owner (tri_words.cu), or one
//    degree-oriented DAG of the union and its out-degree buckets, with a learned
//    schedule installed or where that is faster (batch_tc_plan); a block per graph
//    sums its vertices.
//  * BFS and PageRank of the larger graphs are one cooperative launch each: every
//    level or iteration is one pass over the entries of all of them that are still
//    at work, and the blocks meet at a grid barrier. The entries are read as a
//    stream of 256-entry chunks (8 consecutive entries per lane, a byte per entry
//    says which row it belongs to), so a pass is spread evenly over the GPU
//    whatever the sizes of the graphs. Rows that cross chunks leave parts that are
//    joined after the pass. A small graph is a block's, with one block barrier per
//    level or iteration (batch_small_*).
//  * BFS from S <= 32 sources per graph: multi-source BFS (Then et al., VLDB
//    2015) with one S-bit mask per vertex. A level ORs the neighbours' masks
//    into the vertex's own, from one mask array into another; a bit that is new
//    at level L is distance L. (The masks hold every source seen so far, not
//    the last level's only: an older bit of a neighbour has reached the vertex
//    already.)
//  * Personalised PageRank from K seeds per graph (teleport 1/K per seed,
//    repeats add up; the formula of gcu_personalized_pagerank): every graph
//    iterates to its own convergence (L1 change < tol), FP64 row sums. The change
//    is summed per graph in integers, as a multiple of the tolerance, and the
//    dangling mass in a fixed order, so the result does not depend on which warp
//    did what. Neither has a range: a CSR that is not symmetric, pulled over its
//    own lists, does not conserve mass, nor does a damping outside [0, 1].
// No reference counterpart: the reference runs one graph per call.
#include <algorithm>

#include "device_common.cuh"
#include "gcu_internal.h"

namespace gcu {

constexpr uint32_t kMaxBatchSources = 32;

// ---------------------------------------------------------------- kernels

__global__ void batch_entry_base_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ vbase,
                                        uint32_t G, uint32_t* __restrict__ ebase) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g <= G; g += gridDim.x * blockDim.x)
        ebase[g] = offsets[vbase[g]];
}

// First union entry whose target lies outside its row's graph (atomicMin).
__global__ void batch_check_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets,
                                   const uint32_t* __restrict__ vbase, uint32_t G,
                                   unsigned long long* __restrict__ first_bad) {
    for (uint32_t g = blockIdx.x; g < G; g += gridDim.x) {
        const uint32_t vb = vbase[g], ve = vbase[g + 1];
        const uint32_t e0 = offsets[vb], e1 = offsets[ve];
        for (uint64_t j = static_cast<uint64_t>(e0) + threadIdx.x; j < e1; j += blockDim.x) {
            const uint32_t t = targets[j];
            if (t < vb || t >= ve) atomicMin(first_bad, static_cast<unsigned long long>(j));
        }
    }
}

__global__ void batch_graph_sum_kernel(const unsigned long long* __restrict__ per_vertex,
                                       const uint32_t* __restrict__ vbase, uint32_t G,
                                       unsigned long long* __restrict__ totals) {
    __shared__ unsigned long long scratch[32];
    for (uint32_t g = blockIdx.x; g < G; g += gridDim.x) {
        unsigned long long acc = 0;
        for (uint64_t v = static_cast<uint64_t>(vbase[g]) + threadIdx.x; v < vbase[g + 1]; v += blockDim.x)
            acc += per_vertex[v];
        acc = block_sum(acc, scratch);
        if (threadIdx.x == 0) totals[g] = acc;
    }
}

// Teleport vector: 1/K for every seed (local ids), repeats add up.
__global__ void batch_tele_kernel(const uint32_t* __restrict__ seeds, const uint32_t* __restrict__ vbase, uint32_t G,
                                  uint32_t K, float* __restrict__ tele) {
    const uint64_t total = static_cast<uint64_t>(G) * K;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t g = static_cast<uint32_t>(i / K);
        atomicAdd(tele + vbase[g] + seeds[i], 1.0f / static_cast<float>(K));
    }
}

// Teleport of every seed without entries, 0 for the others (and for kNoSeed).
constexpr uint32_t kNoSeed = 0xFFFFFFFFu;

__global__ void batch_lone_tele_kernel(const uint32_t* __restrict__ seeds, const uint32_t* __restrict__ vbase,
                                       const uint32_t* __restrict__ offsets, const float* __restrict__ tele, uint32_t G,
                                       uint32_t K, float* __restrict__ lone_tele) {
    const uint64_t total = static_cast<uint64_t>(G) * K;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        float p = 0.f;
        if (seeds[i] != kNoSeed) {
            const uint32_t v = vbase[static_cast<uint32_t>(i / K)] + seeds[i];
            if (offsets[v + 1] == offsets[v]) p = tele[v];
        }
        lone_tele[i] = p;
    }
}

// One member graph copied out with local ids.
__global__ void batch_extract_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets,
                                     uint32_t vb, uint32_t n, uint32_t eb, uint32_t m, uint32_t* __restrict__ lo,
                                     uint32_t* __restrict__ lt) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i <= n || i < m;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        if (i <= n) lo[i] = offsets[vb + i] - eb;
        if (i < m) lt[i] = targets[eb + i] - vb;
    }
}

// ---------------------------------------------------------------- passes over the union's entries

constexpr uint32_t kBatchChunk = 256;     // entries per warp step
constexpr int kBatchThreads = 256;
constexpr int kBatchCtasPerSm = 5;
constexpr uint32_t kBatchRun = 2;         // consecutive chunks per warp turn (neighbouring chunks share their graph's lines)
constexpr uint32_t kNone = 0xFFFFFFFFu;

// Graphs of up to this many entries and vertices are a block's (batch_small_*), the
// others take part in the passes over all large graphs. A level of a small graph
// is a few steps of a block and one block barrier, where a pass has a chain of
// dependent loads and two grid barriers, 10 us whatever the graphs' sizes: 8 paths
// of 1,000 vertices, BFS 10.8 -> 0.8 ms, 20 PageRank iterations 0.39 -> 0.11; 600
// graphs of 30,000 entries 0.65 -> 0.21 and 1.75 -> 1.02 ms. Where there are larger
// graphs, the ones of 32,768 to 65,536 entries are better off in their passes than
// in a few blocks of their own afterwards (256 corpus graphs 14.8 against 15.6 ms);
// without, not (16 grids of 40,000 entries, BFS 2.4 against 1.5 ms).
constexpr uint32_t kSmallLimit = 32768, kSmallLimitAlone = 65536;

// Blocks of 1024, 512 or 256 threads. Where the graphs of up to 2,048 or 512 vertices
// are more than twice as many as SMs they have smaller blocks of their own, of which
// more are resident; fewer graphs have the time to themselves, and the largest
// blocks are the fastest.
constexpr int kSmallClasses = 3;
constexpr int kSmallThreads[kSmallClasses] = {1024, 512, 256};
constexpr uint32_t kSmallClassVertices[kSmallClasses] = {kSmallLimitAlone, 2048, 512};

// Measured on one B200, 256 graphs of the generated corpus (6 M vertices, 106 M
// entries), a CTA per graph before: BFS from 16 sources 49.1 -> 3.5 ms (the four
// or five graphs of 4 M entries ran alone at the end), 20 PageRank iterations
// 74.1 -> 6.9 ms (307 G entries/s). Finishing rows in the lanes where they end, one
// after another and their inputs loaded behind the gathers, took 8.0 ms for the
// PageRank (40 registers, 3 x 512 threads). What bounds it now is half issue (57 %
// of the slots), half the L1 (56 %, 44 % hits). CTA shapes, PageRank / BFS: 5 x 256
// threads (48 registers) 6.9 / 3.5 ms, 4 x 256 (64) 7.1 / 3.8, 6 x 256 (40) 7.7 /
// 3.8, 3 x 512 (40) 7.6 / 3.6; turns of 1 / 4 chunks 7.6 / 7.5 ms; a contiguous
// stretch per SM instead of interleaved turns 7.8 / 4.4.

// A large graph, or a small one.
struct BatchGraph {
    uint32_t id;                 // in the batch
    uint32_t v_begin, v_end;     // its vertices,
    uint32_t e_begin, e_end;     // its entries
    uint32_t chunk;              // large: its first chunk
    uint32_t v_before;           // large: vertices of the large graphs before it
};

// What one warp step reads: entries [start, start + kBatchChunk) as far as they are
// the graph's, and the rows that hold them.
struct alignas(16) BatchChunk {
    uint32_t start;   // a multiple of 8 (32-byte loads)
    uint32_t row;     // its first row
    uint32_t graph;   // of the large ones
    uint32_t shape;   // rows | first entry << 9 | end << 12 | first row begun before << 30 | last row goes on << 31
    __device__ __forceinline__ uint32_t rows() const { return shape & 511u; }
    __device__ __forceinline__ uint32_t first() const { return (shape >> 9) & 7u; }
    __device__ __forceinline__ uint32_t end() const { return (shape >> 12) & 511u; }
    __device__ __forceinline__ bool begun_before() const { return (shape >> 30) & 1u; }
    __device__ __forceinline__ bool goes_on() const { return shape >> 31; }
};

// The large graphs' vertices with entries, packed ("rows" below are indices into
// this list), and those without. A graph's chunks are its own.
struct BatchRows {
    const uint32_t* targets;
    const BatchGraph* graphs;
    const uint2* rows;           // (union vertex, entries)
    const BatchChunk* chunks;
    const uint8_t* delta;        // per entry of a chunk: its row minus the chunk's first row
    const uint4* split;          // (row, first chunk, last chunk, graph) of the rows that cross chunks
    const uint2* lone;           // (vertex without entries, graph)
    uint32_t* lists;             // [2][n_chunks]: the chunks of a pass (ChunkList)
    uint32_t n_graphs, n_rows, n_chunks, n_split, n_lone;
};

constexpr uint32_t kMaxLists = 33;
struct BatchRunState {
    GridBarrier bar;
    uint32_t active[3];          // chunks of the graphs at work in this pass (and one per graph), rotating
    uint32_t listed[kMaxLists];  // chunks of each list made
};

// The chunks that a pass goes through: all of them, and once half are of graphs
// that have stopped, a list of the others, made anew each time it has halved. A
// deep graph among large ones is then not charged with theirs: BFS on 121 graphs of
// which one is a path of 20,000 vertices 443 -> 249 ms (a block per graph: 304); a
// whole batch that stops at about the same time 1 % slower to 2 % faster. Not worth
// it below two chunks a warp.
struct ChunkList {  // in shared memory: the passes are short of registers
    const uint32_t* list;  // NULL: chunk i is i
    uint32_t n, made;
};
__device__ __forceinline__ uint32_t list_chunk(const uint32_t* list, uint32_t i) { return list ? list[i] : i; }

__device__ __forceinline__ bool list_halved(const ChunkList& l, uint32_t active) {
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    return l.n > 2 * warps && 2ull * active <= l.n && l.made < kMaxLists;
}

// All threads of the grid, between two barriers; then list_take with the count.
template <class Op>
__device__ __forceinline__ void list_make(const BatchRows& R, const ChunkList& l, const Op& op, BatchRunState* st) {
    uint32_t* to = R.lists + static_cast<size_t>(l.made & 1) * R.n_chunks;
    const uint32_t* from = l.list;
    for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; b < l.n; b += gridDim.x * blockDim.x) {
        const uint32_t i = b + lane_id();
        const uint32_t c = i < l.n ? list_chunk(from, i) : 0u;
        const bool keep = i < l.n && op.works(__ldg(&R.chunks[c].graph));
        const unsigned kept = __ballot_sync(kFullMask, keep);
        uint32_t place = 0;
        if (lane_id() == 0 && kept) place = atomicAdd(st->listed + l.made, static_cast<uint32_t>(__popc(kept)));
        place = __shfl_sync(kFullMask, place, 0) + __popc(kept & ((1u << lane_id()) - 1));
        if (keep) to[place] = c;
    }
}

// By one thread of the block, before a block barrier.
__device__ __forceinline__ void list_take(const BatchRows& R, ChunkList& l, const BatchRunState* st) {
    l.list = R.lists + static_cast<size_t>(l.made & 1) * R.n_chunks;
    l.n = __ldcg(st->listed + l.made);
    ++l.made;
}

__device__ __forceinline__ uint32_t batch_chunk_count(const BatchRows& R, uint64_t g) {
    return (g + 1 < R.n_graphs ? R.graphs[g + 1].chunk : R.n_chunks) - R.graphs[g].chunk;
}

// The last of the graphs that begins at or before x (`first` picks where).
template <class First>
__device__ __forceinline__ uint32_t batch_graph_of(uint32_t n, uint64_t x, First first) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (first(mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// flag[i] = vertex i of the large graphs' (numbered one after the other) has entries.
__global__ void batch_row_flags_kernel(const uint32_t* __restrict__ offsets, const BatchGraph* __restrict__ graphs,
                                       uint32_t n_graphs, uint64_t n, uint32_t* __restrict__ flag) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const BatchGraph& g = graphs[batch_graph_of(n_graphs, i, [&](uint32_t k) { return graphs[k].v_before; })];
        const uint64_t v = g.v_begin + (i - g.v_before);
        flag[i] = offsets[v + 1] > offsets[v] ? 1u : 0u;
    }
}

// Rows and vertices without entries; for each chunk the row of its first and of its
// last entry; whether a row crosses chunks.
__global__ void batch_rows_kernel(const uint32_t* __restrict__ offsets, const BatchGraph* __restrict__ graphs,
                                  uint32_t n_graphs, uint64_t n, const uint32_t* __restrict__ pos,
                                  uint2* __restrict__ rows, uint32_t* __restrict__ row_graph, uint2* __restrict__ lone,
                                  uint32_t* __restrict__ lone_count, uint2* __restrict__ chunk_rows,
                                  uint32_t* __restrict__ split_flag) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t gi = batch_graph_of(n_graphs, i, [&](uint32_t k) { return graphs[k].v_before; });
        const BatchGraph& g = graphs[gi];
        const uint32_t v = g.v_begin + static_cast<uint32_t>(i - g.v_before), r = pos[i];
        if (pos[i + 1] == r) {
            lone[i - r] = make_uint2(v, gi);
            atomicAdd(lone_count + gi, 1u);
            continue;
        }
        const uint32_t s = offsets[v], e = offsets[v + 1], origin = g.e_begin & ~7u;
        const uint32_t c0 = g.chunk + (s - origin) / kBatchChunk, c1 = g.chunk + (e - 1 - origin) / kBatchChunk;
        rows[r] = make_uint2(v, e - s);
        row_graph[r] = gi;
        if (s == g.e_begin || (s - origin) % kBatchChunk == 0) chunk_rows[c0].x = r;
        for (uint32_t c = c0 + 1; c <= c1; ++c) chunk_rows[c].x = r;
        for (uint32_t c = c0; c < c1; ++c) chunk_rows[c].y = r;
        if (e == g.e_end || (e - origin) % kBatchChunk == 0) chunk_rows[c1].y = r;
        split_flag[r] = c0 != c1 ? 1u : 0u;
    }
}

// A warp per chunk: its shape, and each entry's row.
__global__ void __launch_bounds__(256) batch_chunks_kernel(const uint32_t* __restrict__ offsets,
                                                           const BatchGraph* __restrict__ graphs, uint32_t n_graphs,
                                                           uint32_t n_chunks, const uint2* __restrict__ rows,
                                                           const uint2* __restrict__ chunk_rows,
                                                           BatchChunk* __restrict__ chunks,
                                                           uint8_t* __restrict__ delta) {
    const unsigned lane = lane_id();
    for (uint64_t c = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; c < n_chunks;
         c += (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5) {
        const uint32_t gi = batch_graph_of(n_graphs, c, [&](uint32_t k) { return graphs[k].chunk; });
        const BatchGraph& g = graphs[gi];
        const uint32_t start = (g.e_begin & ~7u) + (static_cast<uint32_t>(c) - g.chunk) * kBatchChunk;
        const uint2 r = chunk_rows[c];
        const uint32_t first = start < g.e_begin ? g.e_begin - start : 0u, end = min_u32(kBatchChunk, g.e_end - start);
        if (lane == 0) {
            const bool before = offsets[rows[r.x].x] < start + first;
            const bool on = static_cast<uint64_t>(offsets[rows[r.y].x + 1]) > static_cast<uint64_t>(start) + end;
            chunks[c] = BatchChunk{start, r.x, gi, (r.y - r.x + 1) | first << 9 | end << 12 | (before ? 1u << 30 : 0u) |
                                                       (on ? 1u << 31 : 0u)};
        }
        for (uint32_t i = lane; i < kBatchChunk; i += 32) {
            uint32_t lo = r.x, hi = r.y + 1;  // the last row that begins at or before the entry
            if (i >= first && i < end)
                while (hi - lo > 1) {
                    const uint32_t mid = lo + ((hi - lo) >> 1);
                    if (offsets[rows[mid].x] <= start + i) lo = mid;
                    else hi = mid;
                }
            delta[c * kBatchChunk + i] = static_cast<uint8_t>(lo - r.x);
        }
    }
}

__global__ void batch_split_rows_kernel(const uint32_t* __restrict__ offsets, const BatchGraph* __restrict__ graphs,
                                        uint32_t n_rows, const uint2* __restrict__ rows,
                                        const uint32_t* __restrict__ row_graph, const uint32_t* __restrict__ pos,
                                        uint4* __restrict__ split) {
    for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n_rows;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        if (pos[r + 1] > pos[r]) {
            const BatchGraph& g = graphs[row_graph[r]];
            const uint32_t s = offsets[rows[r].x], origin = g.e_begin & ~7u;
            split[pos[r]] = make_uint4(static_cast<uint32_t>(r), g.chunk + (s - origin) / kBatchChunk,
                                       g.chunk + (s + rows[r].y - 1 - origin) / kBatchChunk, row_graph[r]);
        }
}

// One pass: chunk after chunk, a warp each (kBatchRun consecutive chunks per
// turn), 8 consecutive entries per lane. op gives
//   works(graph)       whether the graph is at work (else its chunks are skipped)
//   enter(graph)       all lanes, before a chunk of it
//   want(vertex)       whether the row's entries have to be gathered
//   gather(target), add(x, y), zero()
//   load(row), more(in)  what finish needs besides the result: loads, and those
//                      that depend on them
//   finish(x, in)      the row's result
//   part(i, x)         part i of a row that crosses chunks: 2c for the end of a row
//                      begun before chunk c, 2c + 1 for a row that goes on after it
//   flush()            after every turn (all lanes)
// Runs of equal rows are joined per lane, then across lanes by a segmented
// scan; the lane where a row ends puts its result into s_row (kBatchChunk of the
// warp's own), from where consecutive lanes finish consecutive rows. The first 32
// rows' inputs are loaded beside the gathers: loads that follow them wait in the
// queue behind them.
template <class Op>
__device__ __forceinline__ void batch_pass(const BatchRows& R, const ChunkList& list, Op& op, typename Op::T* s_row) {
    using T = typename Op::T;
    const unsigned lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    for (uint32_t i0 = warp * kBatchRun; i0 < list.n; i0 += warps * kBatchRun) {  // chunks: far below 2^32
        for (uint32_t ci = i0; ci < min(i0 + kBatchRun, list.n); ++ci) {
            const uint32_t c = list_chunk(list.list, ci);
            const uint4 meta = __ldg(reinterpret_cast<const uint4*>(R.chunks) + c);
            const uint2 dl =
                ld_stream2(reinterpret_cast<const uint2*>(R.delta + static_cast<uint64_t>(c) * kBatchChunk + 8 * lane));
            const BatchChunk k{meta.x, meta.y, meta.z, meta.w};
            if (!op.works(k.graph)) continue;
            op.enter(k.graph);
            uint32_t t[8] = {};
            if (!Op::kSkips && 8 * lane < k.end()) ld_stream8(R.targets + k.start + 8 * lane, t);
            uint32_t row[8];  // less the chunk's first
#pragma unroll
            for (int i = 0; i < 8; ++i)
                row[i] = 8 * lane + i >= k.first() && 8 * lane + i < k.end()
                             ? (((i < 4 ? dl.x : dl.y) >> (8 * (i & 3))) & 0xFFu)
                             : kNone;
            bool want[8];
            bool some = false;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (!Op::kSkips) want[i] = row[i] != kNone;
                else if (i > 0 && row[i] == row[i - 1]) want[i] = want[i - 1];
                else want[i] = row[i] != kNone && op.want(__ldg(&R.rows[k.row + row[i]].x));
                some = some || want[i];
            }
            if (Op::kSkips && some) ld_stream8(R.targets + k.start + 8 * lane, t);
            const uint32_t n_rows = k.rows();
            auto in = op.load(k.row + min(lane, n_rows - 1));
            T val[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) val[i] = op.gather(want[i], t[i]);
            op.more(in);
            T head = Op::zero(), acc = Op::zero();
            bool multi = false;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc = Op::add(acc, val[i]);
                if (i < 7 && row[i + 1] != row[i]) {
                    if (!multi) {
                        head = acc;
                        multi = true;
                    } else {
                        s_row[row[i]] = acc;
                    }
                    acc = Op::zero();
                }
            }
            const uint32_t rf = row[0], rl = row[7];
            const uint32_t prev_last = __shfl_up_sync(kFullMask, rl, 1);
            const uint32_t next_first = __shfl_down_sync(kFullMask, rf, 1);
            const bool carry_in = lane > 0 && prev_last == rf;
            bool head_flag = multi || !carry_in;
            T S = acc;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const T su = __shfl_up_sync(kFullMask, S, d);
                const bool fu = __shfl_up_sync(kFullMask, head_flag, d);
                if (lane >= static_cast<unsigned>(d)) {
                    if (!head_flag) S = Op::add(S, su);
                    head_flag = head_flag || fu;
                }
            }
            const T carry = __shfl_up_sync(kFullMask, S, 1);
            if (multi && rf != kNone) s_row[rf] = carry_in ? Op::add(head, carry) : head;
            const bool continues = lane < 31 && next_first == rl;
            if (!continues && rl != kNone) s_row[rl] = S;  // the last run ends at this lane's end
            __syncwarp();
            for (uint32_t r = lane; r < n_rows; r += 32) {
                if (r >= 32) {
                    in = op.load(k.row + r);
                    op.more(in);
                }
                const T x = s_row[r];
                if (r == n_rows - 1 && k.goes_on()) op.part(2 * static_cast<uint64_t>(c) + 1, x);
                else if (r == 0 && k.begun_before()) op.part(2 * static_cast<uint64_t>(c), x);
                else op.finish(x, in);
            }
            __syncwarp();  // s_row is the next chunk's
        }
        op.flush();
    }
}

// The rows that cross chunks, a thread each: their parts in chunk order.
template <class Op>
__device__ __forceinline__ void batch_split_pass(const BatchRows& R, Op& op) {
    using T = typename Op::T;
    for (uint64_t b = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) & ~31ull; b < R.n_split;
         b += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t i = b + lane_id();
        uint32_t g = kNone;
        if (i < R.n_split) {
            const uint4 s = R.split[i];
            if (op.works(s.w)) {
                g = s.w;
                T x = op.parts(2 * static_cast<uint64_t>(s.y) + 1);
                for (uint32_t c = s.y + 1; c < s.z; ++c) x = Op::add(x, op.parts(2 * static_cast<uint64_t>(c) + 1));
                x = Op::add(x, op.parts(2 * static_cast<uint64_t>(s.z)));
                auto in = op.load(s.x);
                op.set(g);
                op.more(in);
                op.finish(x, in);
            }
        }
        op.flush_lanes(g);
    }
}

// ---------------------------------------------------------------- multi-source BFS

struct BatchBfs {
    BatchRows rows;
    const uint32_t* sources;
    uint32_t V, S, full;
    uint32_t *mask_a, *mask_b;
    uint32_t* parts;
    int32_t* dist;        // NULL: no distances
    uint32_t* fresh;      // [3][graphs]: sources that reached something new, rotating by level
    uint32_t* stop;       // [graphs]: the level a graph stopped before
    uint32_t* reachable;
    int32_t* max_depth;
    BatchRunState* st;
};

__device__ __forceinline__ void batch_label(int32_t* dist, uint32_t V, uint32_t v, uint32_t bits, int32_t level) {
    if (!dist) return;
    for (; bits; bits &= bits - 1) dist[static_cast<uint64_t>(__ffs(bits) - 1) * V + v] = level;
}

struct BfsOp {
    using T = uint32_t;
    static constexpr bool kSkips = true;
    const BatchBfs& a;
    const uint32_t* in;
    uint32_t* out;
    const uint32_t* prev_fresh;  // [graphs], the level before (NULL at level 0)
    uint32_t* fresh;
    uint32_t level;
    uint32_t my_graph = kNone, my_fresh = 0;

    static __device__ __forceinline__ T zero() { return 0u; }
    static __device__ __forceinline__ T add(T x, T y) { return x | y; }
    // A graph works on while the level before found something new.
    __device__ __forceinline__ bool works(uint32_t g) const {
        return a.stop[g] > level && (prev_fresh == nullptr || prev_fresh[g] != 0);
    }
    __device__ __forceinline__ void enter(uint32_t g) {
        if (g != my_graph) flush();
        my_graph = g;
    }
    __device__ __forceinline__ void set(uint32_t) {}
    __device__ __forceinline__ bool want(uint32_t v) const { return in[v] != a.full; }
    __device__ __forceinline__ T gather(bool p, uint32_t t) const { return ld_if(p, in + t, 0u); }
    __device__ __forceinline__ void part(uint64_t i, T x) { a.parts[i] = x; }
    __device__ __forceinline__ T parts(uint64_t i) const { return a.parts[i]; }
    struct In {
        uint32_t v, old;
    };
    __device__ __forceinline__ In load(uint32_t r) const { return In{__ldg(&a.rows.rows[r].x), 0u}; }
    __device__ __forceinline__ void more(In& x) const { x.old = ld_if(true, in + x.v, 0u); }
    __device__ __forceinline__ void finish(T m, const In& x) {
        const uint32_t now = m & ~x.old;
        out[x.v] = x.old | m;
        if (!now) return;
        batch_label(a.dist, a.V, x.v, now, static_cast<int32_t>(level) + 1);
        my_fresh |= now;
    }
    // The warp's graph is the same in all lanes.
    __device__ __forceinline__ void flush() {
        const uint32_t bits = __reduce_or_sync(kFullMask, my_fresh);
        if (bits && lane_id() == 0) atomicOr(fresh + my_graph, bits);
        my_fresh = 0;
    }
    // Each lane has a graph of its own.
    __device__ __forceinline__ void flush_lanes(uint32_t g) {
        if (g != kNone && my_fresh) atomicOr(fresh + g, my_fresh);
        my_fresh = 0;
    }
};

__global__ void __launch_bounds__(kBatchThreads, kBatchCtasPerSm) batch_bfs_kernel(const BatchBfs a) {
    __shared__ uint32_t s_active;
    __shared__ ChunkList s_list;
    if (threadIdx.x == 0) s_list = ChunkList{nullptr, a.rows.n_chunks, 0};  // before the first barrier
    __shared__ uint32_t s_count[kMaxBatchSources];
    __shared__ uint32_t s_rows[kBatchThreads / 32][kBatchChunk];
    const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t nthreads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint32_t G = a.rows.n_graphs;
    unsigned barriers = 0;
    for (uint64_t r = tid; r < a.rows.n_rows; r += nthreads) {
        const uint32_t v = a.rows.rows[r].x;
        a.mask_a[v] = 0;
        a.mask_b[v] = 0;
    }
    for (uint64_t i = tid; i < a.rows.n_lone; i += nthreads) {
        const uint32_t v = a.rows.lone[i].x;
        a.mask_a[v] = 0;
        a.mask_b[v] = 0;
    }
    for (uint64_t g = tid; g < G; g += nthreads) {
        for (int q = 0; q < 3; ++q) a.fresh[static_cast<uint64_t>(q) * G + g] = 0;
        a.stop[g] = kNone;
        for (uint32_t k = 0; k < a.S; ++k) a.max_depth[static_cast<uint64_t>(a.rows.graphs[g].id) * a.S + k] = 0;
    }
    if (!grid_barrier(&a.st->bar, barriers)) return;
    for (uint64_t i = tid; i < static_cast<uint64_t>(G) * a.S; i += nthreads) {
        const BatchGraph& g = a.rows.graphs[i / a.S];
        const uint32_t k = static_cast<uint32_t>(i % a.S);
        const uint32_t v = g.v_begin + a.sources[static_cast<uint64_t>(g.id) * a.S + k];
        // Both arrays: a vertex without entries is never written again.
        atomicOr(a.mask_a + v, 1u << k);
        atomicOr(a.mask_b + v, 1u << k);
        if (a.dist) a.dist[static_cast<uint64_t>(k) * a.V + v] = 0;
    }
    if (!grid_barrier(&a.st->bar, barriers)) return;
    // Each level labels something in some graph, or is the last.
    for (uint32_t level = 0;; ++level) {
        BfsOp op{a, (level & 1) ? a.mask_b : a.mask_a, (level & 1) ? a.mask_a : a.mask_b,
                 level ? a.fresh + static_cast<uint64_t>((level + 2) % 3) * G : nullptr,
                 a.fresh + static_cast<uint64_t>(level % 3) * G, level};
        for (uint64_t g = tid; g < G; g += nthreads) {
            a.fresh[static_cast<uint64_t>((level + 1) % 3) * G + g] = 0;  // last read a level ago
            if (a.stop[g] <= level) continue;
            if (level) {
                uint32_t bits = op.prev_fresh[g];
                if (!bits) {
                    a.stop[g] = level;
                    continue;
                }
                const uint64_t base = static_cast<uint64_t>(a.rows.graphs[g].id) * a.S;
                for (; bits; bits &= bits - 1) a.max_depth[base + __ffs(bits) - 1] = static_cast<int32_t>(level);
            }
            atomicAdd(a.st->active + level % 3, 1u + batch_chunk_count(a.rows, g));
        }
        if (tid == 0) a.st->active[(level + 1) % 3] = 0;
        batch_pass(a.rows, s_list, op, s_rows[threadIdx.x >> 5]);
        if (!grid_barrier(&a.st->bar, gridDim.x, barriers, [&] { s_active = __ldcg(a.st->active + level % 3); })) return;
        if (s_active == 0) break;
        const bool halved = list_halved(s_list, s_active);
        if (halved) list_make(a.rows, s_list, op, a.st);
        batch_split_pass(a.rows, op);
        if (!grid_barrier(&a.st->bar, gridDim.x, barriers, [&] { if (halved) list_take(a.rows, s_list, a.st); })) return;
    }
    // Reached vertices per source: lane k of every warp counts bit k of its
    // graph's vertices. A graph that has stopped has the same masks in both arrays.
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    for (uint32_t i = blockIdx.x; i < G; i += gridDim.x) {
        const BatchGraph& g = a.rows.graphs[i];
        if (threadIdx.x < kMaxBatchSources) s_count[threadIdx.x] = 0;
        __syncthreads();
        uint32_t cnt = 0;
        for (uint64_t base = static_cast<uint64_t>(g.v_begin) + warp * 32; base < g.v_end; base += kBatchThreads) {
            const uint64_t v = base + lane;
            const uint32_t vis = v < g.v_end ? a.mask_a[v] : 0u;
            for (uint32_t k = 0; k < a.S; ++k) {
                const unsigned b = __ballot_sync(kFullMask, (vis >> k) & 1u);
                if (lane == k) cnt += __popc(b);
            }
        }
        if (lane < a.S && cnt) atomicAdd(&s_count[lane], cnt);
        __syncthreads();
        if (threadIdx.x < a.S) a.reachable[static_cast<uint64_t>(g.id) * a.S + threadIdx.x] = s_count[threadIdx.x];
        __syncthreads();
    }
}

// ---------------------------------------------------------------- personalised PageRank

// A graph's L1 change, of which only whether it is below the tolerance is asked:
// the sum of the warps' parts in units of 2^-62 of the tolerance, the low 32 bits
// of each part in one word and the rest in the other, so that no sum of 2^32 parts
// overflows. A part that is not below the tolerance itself (NaN, or any part where
// the tolerance is not positive) counts as twice the tolerance.
struct alignas(16) ChangeSum {
    unsigned long long low, high;
};
constexpr double kChangeUnits = 4611686018427387904.0;  // 2^62
constexpr unsigned long long kChangeLimit = 1ull << 30;  // of the high parts

__device__ __forceinline__ void add_change(ChangeSum* sum, double part, double tolerance, double scale) {
    if (!(part < tolerance)) {
        atomicAdd(&sum->high, 2 * kChangeLimit);
    } else if (const unsigned long long q = __double2ull_rz(part * scale)) {
        if (q & 0xFFFFFFFFull) atomicAdd(&sum->low, q & 0xFFFFFFFFull);
        if (q >> 32) atomicAdd(&sum->high, q >> 32);
    }
}
__device__ __forceinline__ bool below_tolerance(const ChangeSum& c) { return c.high + (c.low >> 32) < kChangeLimit; }

// A vertex's new rank from the contributions of its entries, its teleport and its
// graph's dangling mass.
__device__ __forceinline__ float batch_rank(double damp, double sum, double tele, double mass) {
    return static_cast<float>((1.0 - damp) * tele + damp * (sum + mass * tele));
}

struct BatchPpr {
    BatchRows rows;
    const uint32_t* lone_count;  // [graphs]
    const float* tele;
    const float* lone_tele;      // [G][K] of the seeds without entries (each once), 0 for the others
    uint32_t K, log_lanes;       // 2^log_lanes lanes sum a graph's dangling mass
    double damp, tolerance, scale;
    uint32_t max_iterations;
    float *contrib_a, *contrib_b;
    float* ranks;
    double* parts;
    ChangeSum* change;           // [3][graphs], rotating by iteration
    double* mass;                // [2][graphs]: dangling mass, alternating
    uint32_t* stop;              // [graphs]: iterations a graph has run when it stopped
    uint32_t* iterations;
    uint8_t* converged;
    BatchRunState* st;
};

struct PprOp {
    using T = double;
    static constexpr bool kSkips = false;
    const BatchPpr& a;
    const float* in;
    float* out;
    const ChangeSum* prev_change;  // [graphs], the iteration before
    const double* mass;            // [graphs]
    ChangeSum* change;
    uint32_t it;
    uint32_t my_graph = kNone;
    double my_mass = 0.0, my_change = 0.0;

    static __device__ __forceinline__ T zero() { return 0.0; }
    static __device__ __forceinline__ T add(T x, T y) { return x + y; }
    __device__ __forceinline__ bool works(uint32_t g) const {
        return a.stop[g] > it && (it == 0 || !below_tolerance(prev_change[g]));
    }
    __device__ __forceinline__ void enter(uint32_t g) {
        if (g == my_graph) return;
        flush();
        my_graph = g;
        my_mass = mass[g];
    }
    __device__ __forceinline__ void set(uint32_t g) { my_mass = mass[g]; }
    __device__ __forceinline__ bool want(uint32_t) const { return true; }
    __device__ __forceinline__ T gather(bool p, uint32_t t) const {
        return static_cast<double>(__uint_as_float(ld_if(p, reinterpret_cast<const uint32_t*>(in) + t, 0u)));
    }
    __device__ __forceinline__ void part(uint64_t i, T x) { a.parts[i] = x; }
    __device__ __forceinline__ T parts(uint64_t i) const { return a.parts[i]; }
    __device__ __forceinline__ float update(uint32_t v, double sum, float tele, float old) {
        const float x = batch_rank(a.damp, sum, static_cast<double>(tele), my_mass);
        my_change += fabs(static_cast<double>(x) - static_cast<double>(old));
        a.ranks[v] = x;
        return x;
    }
    struct In {
        uint32_t v, len;
        float tele, old;
    };
    __device__ __forceinline__ In load(uint32_t r) const {
        const uint2 row = __ldg(a.rows.rows + r);
        return In{row.x, row.y, 0.f, 0.f};
    }
    __device__ __forceinline__ void more(In& x) const {
        x.tele = __ldg(a.tele + x.v);
        x.old = __uint_as_float(ld_if(true, reinterpret_cast<const uint32_t*>(a.ranks) + x.v, 0u));
    }
    __device__ __forceinline__ void finish(T sum, const In& in) {
        out[in.v] = update(in.v, sum, in.tele, in.old) / static_cast<float>(in.len);
    }
    // The warp's graph is the same in all lanes.
    __device__ __forceinline__ void flush() {
        if (my_graph != kNone) {
            const double part = warp_sum(my_change);
            if (lane_id() == 0) add_change(change + my_graph, part, a.tolerance, a.scale);
            my_change = 0.0;
        }
        my_graph = kNone;
    }
    // Each lane has a graph of its own (kNone: none); one for all lanes nearly always.
    __device__ __forceinline__ void flush_lanes(uint32_t g) {
        const unsigned has = __ballot_sync(kFullMask, g != kNone);
        if (has) {
            const uint32_t g0 = __shfl_sync(kFullMask, g, __ffs(has) - 1);
            const double part = warp_sum(g == g0 ? my_change : 0.0);
            if (lane_id() == static_cast<unsigned>(__ffs(has) - 1)) add_change(change + g0, part, a.tolerance, a.scale);
            if (g != g0 && g != kNone) add_change(change + g, my_change, a.tolerance, a.scale);
        }
        my_change = 0.0;
    }
};

// The dangling mass of the ranks that an iteration makes from the mass before it: a
// vertex without entries gets nothing but its teleport, so its rank follows from
// that mass alone, and is 0 unless it is a seed. A group of lanes per graph, in a
// fixed order.
__device__ __forceinline__ void batch_next_mass(const BatchPpr& a, const double* mass, double* next, uint64_t tid,
                                                uint64_t nthreads) {
    const uint32_t lanes = 1u << a.log_lanes, at = static_cast<uint32_t>(tid) & (lanes - 1);
    for (uint64_t b = (tid & ~31ull) >> a.log_lanes; b < a.rows.n_graphs; b += nthreads >> a.log_lanes) {
        const uint64_t g = b + (lane_id() >> a.log_lanes);
        double sum = 0.0;
        if (g < a.rows.n_graphs) {
            const double m = mass[g];
            const float* tele = a.lone_tele + static_cast<uint64_t>(a.rows.graphs[g].id) * a.K;
            for (uint32_t k = at; k < a.K; k += lanes) {
                const float p = __ldg(tele + k);
                if (p != 0.f) sum += static_cast<double>(batch_rank(a.damp, 0.0, static_cast<double>(p), m));
            }
            // The others' rank is 0, or NaN once the mass is no number.
            if (at == 0 && a.lone_count[g] > 0) sum += static_cast<double>(batch_rank(a.damp, 0.0, 0.0, m));
        }
        for (uint32_t d = lanes / 2; d > 0; d /= 2) sum += __shfl_xor_sync(kFullMask, sum, d);
        if (g < a.rows.n_graphs && at == 0) next[g] = sum;
    }
}

__global__ void __launch_bounds__(kBatchThreads, kBatchCtasPerSm) batch_ppr_kernel(const BatchPpr a) {
    __shared__ uint32_t s_active;
    __shared__ ChunkList s_list;
    if (threadIdx.x == 0) s_list = ChunkList{nullptr, a.rows.n_chunks, 0};  // before the first barrier
    __shared__ double s_rows[kBatchThreads / 32][kBatchChunk];
    const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t nthreads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint32_t G = a.rows.n_graphs;
    unsigned barriers = 0;
    auto start = [&](uint32_t g) { return 1.0f / static_cast<float>(a.rows.graphs[g].v_end - a.rows.graphs[g].v_begin); };
    for (uint64_t c = tid >> 5; c < a.rows.n_chunks; c += nthreads >> 5) {
        const BatchChunk k = a.rows.chunks[c];
        const float r0 = start(k.graph);
        for (uint32_t r = lane_id(); r < k.rows(); r += 32) {
            if (r == 0 && k.begun_before()) continue;
            const uint2 row = a.rows.rows[k.row + r];
            a.ranks[row.x] = r0;
            a.contrib_a[row.x] = r0 / static_cast<float>(row.y);
        }
    }
    for (uint64_t i = tid; i < a.rows.n_lone; i += nthreads) {
        // A CSR that is not symmetric may list such a vertex as a target.
        const uint2 v = a.rows.lone[i];
        a.ranks[v.x] = start(v.y);
        a.contrib_a[v.x] = 0.f;
        a.contrib_b[v.x] = 0.f;
    }
    for (uint64_t g = tid; g < G; g += nthreads) {
        for (uint64_t q = 0; q < 3; ++q) a.change[q * G + g] = ChangeSum{0, 0};
        a.mass[g] = static_cast<double>(a.lone_count[g]) * static_cast<double>(start(static_cast<uint32_t>(g)));
        a.stop[g] = kNone;
    }
    if (!grid_barrier(&a.st->bar, barriers)) return;
    for (uint32_t it = 0; it < a.max_iterations; ++it) {
        const uint64_t cur = static_cast<uint64_t>(it % 3) * G, prev = static_cast<uint64_t>((it + 2) % 3) * G;
        const uint64_t next = static_cast<uint64_t>((it + 1) % 3) * G;
        PprOp op{a, (it & 1) ? a.contrib_b : a.contrib_a, (it & 1) ? a.contrib_a : a.contrib_b,
                 a.change + prev, a.mass + static_cast<uint64_t>(it & 1) * G, a.change + cur, it};
        for (uint64_t g = tid; g < G; g += nthreads) {
            a.change[next + g] = ChangeSum{0, 0};  // last read an iteration ago
            if (a.stop[g] <= it) continue;
            if (it && below_tolerance(op.prev_change[g])) a.stop[g] = it;
            else atomicAdd(a.st->active + it % 3, 1u + batch_chunk_count(a.rows, g));
        }
        batch_next_mass(a, op.mass, a.mass + static_cast<uint64_t>(~it & 1) * G, tid, nthreads);
        if (tid == 0) a.st->active[(it + 1) % 3] = 0;
        for (uint64_t b = tid & ~31ull; b < a.rows.n_lone; b += nthreads) {
            uint32_t g = kNone;
            if (b + lane_id() < a.rows.n_lone) {
                const uint2 v = __ldg(a.rows.lone + b + lane_id());
                if (op.works(v.y)) {
                    g = v.y;
                    op.set(g);
                    op.update(v.x, 0.0, a.tele[v.x], a.ranks[v.x]);
                }
            }
            op.flush_lanes(g);
        }
        batch_pass(a.rows, s_list, op, s_rows[threadIdx.x >> 5]);
        if (!grid_barrier(&a.st->bar, gridDim.x, barriers, [&] { s_active = __ldcg(a.st->active + it % 3); })) return;
        if (s_active == 0) break;
        const bool halved = list_halved(s_list, s_active);
        if (halved) list_make(a.rows, s_list, op, a.st);
        batch_split_pass(a.rows, op);
        if (!grid_barrier(&a.st->bar, gridDim.x, barriers, [&] { if (halved) list_take(a.rows, s_list, a.st); })) return;
    }
    // A graph whose last iteration met the tolerance has not been marked yet.
    for (uint64_t g = tid; g < G; g += nthreads) {
        uint32_t n = a.stop[g];
        bool conv = n != kNone;
        if (!conv) {
            n = a.max_iterations;
            conv = n > 0 && below_tolerance(a.change[static_cast<uint64_t>((n + 2) % 3) * G + g]);
        }
        a.iterations[a.rows.graphs[g].id] = n;
        a.converged[a.rows.graphs[g].id] = conv ? 1 : 0;
    }
}

// ---------------------------------------------------------------- small graphs: a block each

// The small graphs, largest first; a block takes the next one when it is done. A
// row of up to kSoloRow entries is a lane's, a longer one its warp's. The walks
// count from a graph's first vertex and a row's first entry: a union may end
// within a block's step of 2^32 vertices or entries.
struct BatchSmall {
    const uint32_t* offsets;
    const uint32_t* targets;
    const BatchGraph* graphs;
    uint32_t n_graphs;
    uint32_t* next;
};
constexpr uint32_t kSoloRow = 31;

// f(graph) for the graphs that this block takes.
template <class F>
__device__ __forceinline__ void for_each_small(const BatchSmall& s, F f) {
    __shared__ uint32_t s_item;
    while (true) {
        if (threadIdx.x == 0) s_item = atomicAdd(s.next, 1u);
        __syncthreads();
        const uint32_t i = s_item;
        if (i >= s.n_graphs) break;
        f(s.graphs[i]);
        __syncthreads();  // s_item, and what f keeps in shared memory
    }
}

struct BatchSmallBfs {
    BatchSmall small;
    const uint32_t* sources;
    uint32_t V, S, full;
    uint32_t *mask_a, *mask_b;
    int32_t* dist;
    uint32_t* reachable;
    int32_t* max_depth;
};

template <int kThreads>
__global__ void __launch_bounds__(kThreads) batch_small_bfs_kernel(const BatchSmallBfs a) {
    constexpr int kWarps = kThreads / 32;
    __shared__ uint32_t s_fresh[2][kWarps];
    __shared__ uint32_t s_count[kMaxBatchSources];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    for_each_small(a.small, [&](const BatchGraph& g) {
        const uint64_t base = static_cast<uint64_t>(g.id) * a.S;
        const uint32_t n = g.v_end - g.v_begin;
        for (uint32_t i = threadIdx.x; i < n; i += kThreads) a.mask_a[g.v_begin + i] = 0;
        if (threadIdx.x < kMaxBatchSources) s_count[threadIdx.x] = 0;
        __syncthreads();
        if (threadIdx.x < a.S) {
            const uint32_t v = g.v_begin + a.sources[base + threadIdx.x];
            atomicOr(a.mask_a + v, 1u << threadIdx.x);
            if (a.dist) a.dist[static_cast<uint64_t>(threadIdx.x) * a.V + v] = 0;
        }
        __syncthreads();
        uint32_t* in = a.mask_a;
        uint32_t* out = a.mask_b;
        int32_t depth = 0;  // of source threadIdx.x
        for (int32_t level = 0;; ++level) {
            uint32_t fresh = 0;
            for (uint32_t b = warp * 32; b < n; b += kThreads) {
                const bool real = b + lane < n;
                const uint32_t v = g.v_begin + b + lane;
                uint32_t old = a.full, s = 0, e = 0;
                if (real) {
                    old = in[v];
                    s = __ldg(a.small.offsets + v);
                    e = __ldg(a.small.offsets + v + 1);
                }
                uint32_t m = 0;
                const bool open = old != a.full;
                if (open && e - s <= kSoloRow)
                    for (uint32_t j = s; j < e && (m | old) != a.full; ++j) m |= in[__ldg(a.small.targets + j)];
                for (unsigned longs = __ballot_sync(kFullMask, open && e - s > kSoloRow); longs; longs &= longs - 1) {
                    const int l = __ffs(longs) - 1;
                    const uint32_t len = __shfl_sync(kFullMask, e - s, l);
                    const uint32_t* list = a.small.targets + __shfl_sync(kFullMask, s, l);
                    const uint32_t lold = __shfl_sync(kFullMask, old, l);
                    uint32_t got = 0;
                    for (uint32_t o = lane; o - lane < len && (got | lold) != a.full; o += 64) {
                        uint32_t x = o < len ? in[__ldg(list + o)] : 0u;
                        if (o + 32 < len) x |= in[__ldg(list + o + 32)];
                        got |= __reduce_or_sync(kFullMask, x);
                    }
                    if (static_cast<int>(lane) == l) m = got;
                }
                if (real) {
                    const uint32_t now = m & ~old;
                    out[v] = old | m;
                    batch_label(a.dist, a.V, v, now, level + 1);
                    fresh |= now;
                }
            }
            // The levels' words alternate, so one barrier a level does.
            fresh = __reduce_or_sync(kFullMask, fresh);
            if (lane == 0) s_fresh[level & 1][warp] = fresh;
            __syncthreads();
            const uint32_t all = __reduce_or_sync(kFullMask, lane < kWarps ? s_fresh[level & 1][lane] : 0u);
            uint32_t* t = in;
            in = out;
            out = t;
            if (all == 0) break;
            if (threadIdx.x < a.S && ((all >> threadIdx.x) & 1u)) depth = level + 1;
        }
        // Reached vertices per source: lane k of every warp counts bit k.
        uint32_t cnt = 0;
        for (uint32_t b = warp * 32; b < n; b += kThreads) {
            const uint32_t vis = b + lane < n ? in[g.v_begin + b + lane] : 0u;
            for (uint32_t k = 0; k < a.S; ++k) {
                const unsigned some = __ballot_sync(kFullMask, (vis >> k) & 1u);
                if (lane == k) cnt += __popc(some);
            }
        }
        if (lane < a.S && cnt) atomicAdd(&s_count[lane], cnt);
        __syncthreads();
        if (threadIdx.x < a.S) {
            a.reachable[base + threadIdx.x] = s_count[threadIdx.x];
            a.max_depth[base + threadIdx.x] = depth;
        }
    });
}

// sum + the contributions of entries o, o + stride, ... of a list, in that order,
// kLoads of them in flight.
template <int kLoads>
__device__ __forceinline__ double add_entries(double sum, const uint32_t* list, const float* in, uint32_t o,
                                              uint32_t stride, uint32_t len) {
    uint32_t x[kLoads];
#pragma unroll
    for (int q = 0; q < kLoads; ++q) x[q] = ld_nc_if(o + q * stride < len, list + o + q * stride, 0u);
#pragma unroll
    for (int q = 0; q < kLoads; ++q)
        x[q] = ld_if(o + q * stride < len, reinterpret_cast<const uint32_t*>(in) + x[q], 0u);
#pragma unroll
    for (int q = 0; q < kLoads; ++q) sum += static_cast<double>(__uint_as_float(x[q]));
    return sum;
}
constexpr int kSoloLoads = 4, kWarpLoads = 8;

struct BatchSmallPpr {
    BatchSmall small;
    const float* tele;
    double damp, tolerance;
    uint32_t max_iterations;
    float *contrib_a, *contrib_b;
    float* ranks;
    uint32_t* iterations;
    uint8_t* converged;
};

template <int kThreads>
__global__ void __launch_bounds__(kThreads) batch_small_ppr_kernel(const BatchSmallPpr a) {
    constexpr int kWarps = kThreads / 32;
    __shared__ double s_sums[2][2][kWarps];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    unsigned parity = 0;
    // Both sums over the block, in a fixed order; the words alternate, so one barrier does.
    auto block_sums = [&](double& x, double& y) {
        x = warp_sum(x);
        y = warp_sum(y);
        if (lane == 0) {
            s_sums[parity][0][warp] = x;
            s_sums[parity][1][warp] = y;
        }
        __syncthreads();
        x = warp_sum(lane < kWarps ? s_sums[parity][0][lane] : 0.0);
        y = warp_sum(lane < kWarps ? s_sums[parity][1][lane] : 0.0);
        parity ^= 1u;
    };
    for_each_small(a.small, [&](const BatchGraph& g) {
        const uint32_t n = g.v_end - g.v_begin;
        const float r0 = 1.0f / static_cast<float>(n);
        double mass = 0.0, change = 0.0;
        for (uint32_t i = threadIdx.x; i < n; i += kThreads) {
            const uint32_t v = g.v_begin + i;
            const uint32_t deg = __ldg(a.small.offsets + v + 1) - __ldg(a.small.offsets + v);
            a.ranks[v] = r0;
            a.contrib_a[v] = deg ? r0 / static_cast<float>(deg) : 0.f;
            if (!deg) mass += static_cast<double>(r0);
        }
        block_sums(change, mass);
        const float* in = a.contrib_a;
        float* out = a.contrib_b;
        uint32_t it = 0;
        bool conv = n == 0;
        while (!conv && it < a.max_iterations) {
            double dangling = 0.0;
            change = 0.0;
            for (uint32_t b = warp * 32; b < n; b += kThreads) {
                const bool real = b + lane < n;
                const uint32_t v = g.v_begin + b + lane;
                uint32_t s = 0, e = 0;
                float tele = 0.f, old = 0.f;
                if (real) {
                    s = __ldg(a.small.offsets + v);
                    e = __ldg(a.small.offsets + v + 1);
                    tele = __ldg(a.tele + v);
                    old = a.ranks[v];
                }
                double sum = 0.0;
                if (e - s <= kSoloRow)
                    for (uint32_t o = 0; o < e - s; o += kSoloLoads)
                        sum = add_entries<kSoloLoads>(sum, a.small.targets + s, in, o, 1, e - s);
                for (unsigned longs = __ballot_sync(kFullMask, e - s > kSoloRow); longs; longs &= longs - 1) {
                    const int l = __ffs(longs) - 1;
                    const uint32_t len = __shfl_sync(kFullMask, e - s, l);
                    const uint32_t* list = a.small.targets + __shfl_sync(kFullMask, s, l);
                    double part = 0.0;
                    for (uint32_t o = lane; o < len; o += 32 * kWarpLoads)
                        part = add_entries<kWarpLoads>(part, list, in, o, 32, len);
                    part = warp_sum(part);
                    if (static_cast<int>(lane) == l) sum = part;
                }
                if (real) {
                    const float x = batch_rank(a.damp, sum, static_cast<double>(tele), mass);
                    change += fabs(static_cast<double>(x) - static_cast<double>(old));
                    a.ranks[v] = x;
                    out[v] = e > s ? x / static_cast<float>(e - s) : 0.f;
                    if (e == s) dangling += static_cast<double>(x);
                }
            }
            block_sums(change, dangling);
            mass = dangling;
            float* t = const_cast<float*>(in);
            in = out;
            out = t;
            ++it;
            conv = change < a.tolerance;
        }
        if (threadIdx.x == 0) {
            a.iterations[g.id] = it;
            a.converged[g.id] = conv ? 1 : 0;
        }
    });
}

// ---------------------------------------------------------------- host

struct BatchImpl {
    std::shared_ptr<DeviceImpl> dev;
    GraphImpl u;  // the union CSR
    uint32_t G = 0;
    std::vector<uint32_t> vbase, ebase;
    DeviceBuffer<uint32_t> d_vbase;
    // Of the BFS and PageRank (built when the first sources or seeds are set).
    bool parted = false;
    BatchRows rows{};
    DeviceBuffer<BatchGraph> large, small;
    DeviceBuffer<uint2> row_list, lone;
    DeviceBuffer<BatchChunk> chunks;
    DeviceBuffer<uint32_t> lone_count, chunk_lists, next_small;
    DeviceBuffer<uint8_t> delta;
    DeviceBuffer<uint4> split;
    uint32_t n_small[kSmallClasses] = {};  // by block size
    DeviceBuffer<BatchRunState> bfs_state, ppr_state;
    unsigned bfs_grid = 0, ppr_grid = 0;
    BatchTcPlan* tc = nullptr;
    std::string tc_tuning;
    DeviceBuffer<unsigned long long> tri_vertex, tri_totals;
    // BFS
    uint32_t S = 0;
    bool keep_dist = true;
    bool bfs_timed = false;
    DeviceBuffer<uint32_t> sources, mask_a, mask_b, bfs_parts, fresh, bfs_stop, reachable;
    DeviceBuffer<int32_t> dist, max_depth;
    // personalised PageRank
    uint32_t K = 0;
    float damping = 0.85f, tolerance = 1e-6f;
    uint32_t max_iterations = 100;
    bool ppr_timed = false;
    DeviceBuffer<uint32_t> seeds, iterations, ppr_stop;
    DeviceBuffer<uint8_t> converged;
    DeviceBuffer<float> tele, lone_tele, contrib_a, contrib_b, ranks;
    DeviceBuffer<double> ppr_parts, mass;
    DeviceBuffer<ChangeSum> change;
    // captured replay of the three
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::string bfs_tuning, ppr_tuning;

    ~BatchImpl() {
        if (dev) dev->activate();
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        destroy_batch_tc_plan(tc);
    }
};

void destroy_batch(BatchImpl* b) { delete b; }

namespace {

uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

unsigned small_grid(const DeviceImpl& dev, uint64_t n, unsigned threads) {
    return static_cast<unsigned>(
        std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(n, threads), static_cast<uint64_t>(dev.sm_count) * 8)));
}

// vbase uploaded, ebase gathered.
Error finish_layout(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    const uint32_t G = b.G;
    GCU_TRY(b.d_vbase.allocate(dev, G + 1));
    GCU_CUDA(cudaMemcpyAsync(b.d_vbase.ptr, b.vbase.data(), 4 * (G + 1), cudaMemcpyHostToDevice, dev.stream), "copy");
    DeviceBuffer<uint32_t> d_ebase;
    GCU_TRY(d_ebase.allocate(dev, G + 1));
    GCU_LAUNCH(dev, "batch_entry_base", batch_entry_base_kernel, small_grid(dev, G + 1, 256), 256, 0, b.u.offsets.ptr,
               b.d_vbase.ptr, G, d_ebase.ptr);
    b.ebase.resize(G + 1);
    GCU_CUDA(cudaMemcpyAsync(b.ebase.data(), d_ebase.ptr, 4 * (G + 1), cudaMemcpyDeviceToHost, dev.stream), "copy");
    // Zero until a pass kernel runs: results may be read before.
    for (auto* st : {&b.bfs_state, &b.ppr_state}) {
        GCU_TRY(st->allocate(dev, 1));
        GCU_CUDA(cudaMemsetAsync(st->ptr, 0, sizeof(BatchRunState), dev.stream), "memset");
    }
    return dev.sync();
}

uint32_t source_bits(const BatchImpl& b) { return b.S >= 32 ? 0xFFFFFFFFu : (1u << b.S) - 1u; }

Error upload(DeviceImpl& dev, const std::vector<BatchGraph>& list, DeviceBuffer<BatchGraph>* to) {
    GCU_TRY(to->allocate(dev, list.size()));
    if (!list.empty())
        GCU_CUDA(cudaMemcpyAsync(to->ptr, list.data(), sizeof(BatchGraph) * list.size(), cudaMemcpyHostToDevice,
                                 dev.stream),
                 "copy");
    return ok();
}

// The small graphs, largest first, and the rows and chunks of the large ones.
Error part_graphs(BatchImpl& b) {
    if (b.parted) return ok();
    DeviceImpl& dev = *b.dev;
    std::vector<BatchGraph> small, large;
    uint64_t n_chunks = 0, n_vertices = 0;
    uint32_t limit = kSmallLimitAlone;
    for (uint32_t i = 0; i < b.G; ++i)
        if (std::max(b.ebase[i + 1] - b.ebase[i], b.vbase[i + 1] - b.vbase[i]) > kSmallLimitAlone) limit = kSmallLimit;
    for (uint32_t i = 0; i < b.G; ++i) {
        BatchGraph g{i, b.vbase[i], b.vbase[i + 1], b.ebase[i], b.ebase[i + 1], 0, 0};
        const uint32_t entries = g.e_end - g.e_begin, vertices = g.v_end - g.v_begin;
        if (std::max(entries, vertices) <= limit) {
            small.push_back(g);
            continue;
        }
        g.chunk = static_cast<uint32_t>(n_chunks);
        g.v_before = static_cast<uint32_t>(n_vertices);
        large.push_back(g);
        n_vertices += vertices;
        if (entries) n_chunks += ceil_div_u64(g.e_end - (g.e_begin & ~7u), kBatchChunk);
    }
    // By class, and largest first in each. A class with few graphs joins the one before.
    auto class_of = [](const BatchGraph& g) {
        int c = 0;
        while (c + 1 < kSmallClasses && g.v_end - g.v_begin <= kSmallClassVertices[c + 1]) ++c;
        return c;
    };
    std::fill(b.n_small, b.n_small + kSmallClasses, 0u);
    for (const BatchGraph& g : small) ++b.n_small[class_of(g)];
    int joins[kSmallClasses] = {};
    for (int c = 1; c < kSmallClasses; ++c) {
        joins[c] = b.n_small[c] > 2u * static_cast<uint32_t>(dev.sm_count) ? c : joins[c - 1];
        if (joins[c] != c) {
            b.n_small[joins[c]] += b.n_small[c];
            b.n_small[c] = 0;
        }
    }
    // Warps beyond a graph's vertices have nothing to do: a class whose graphs are all
    // that small has smaller blocks, unless those have graphs of their own.
    uint32_t widest[kSmallClasses] = {};
    for (const BatchGraph& g : small) {
        uint32_t& w = widest[joins[class_of(g)]];
        w = std::max(w, g.v_end - g.v_begin);
    }
    for (int c = 0; c + 1 < kSmallClasses; ++c)
        for (int k = kSmallClasses - 1; k > c && b.n_small[c]; --k)
            if (!b.n_small[k] && widest[c] <= static_cast<uint32_t>(kSmallThreads[k])) {
                std::swap(b.n_small[c], b.n_small[k]);
                for (int& j : joins)
                    if (j == c) j = k;
            }
    std::stable_sort(small.begin(), small.end(), [&](const BatchGraph& x, const BatchGraph& y) {
        const int cx = joins[class_of(x)], cy = joins[class_of(y)];
        return cx != cy ? cx < cy : x.e_end - x.e_begin > y.e_end - y.e_begin;
    });
    GCU_TRY(upload(dev, small, &b.small));
    GCU_TRY(upload(dev, large, &b.large));
    GCU_TRY(b.next_small.allocate(dev, 2 * kSmallClasses));
    const uint32_t n_graphs = static_cast<uint32_t>(large.size());
    b.rows = BatchRows{};
    GCU_TRY(b.lone_count.allocate(dev, n_graphs));
    if (n_graphs) {
        DeviceBuffer<uint32_t> pos, row_graph, split_pos;
        DeviceBuffer<uint2> chunk_rows;
        GCU_TRY(pos.allocate(dev, n_vertices + 1));
        GCU_LAUNCH(dev, "batch_row_flags", batch_row_flags_kernel, small_grid(dev, n_vertices, 256), 256, 0,
                   b.u.offsets.ptr, b.large.ptr, n_graphs, n_vertices, pos.ptr);
        GCU_TRY(exclusive_scan_u32(dev, pos.ptr, pos.ptr, n_vertices));
        uint32_t n_rows = 0, n_split = 0;
        GCU_CUDA(cudaMemcpyAsync(&n_rows, pos.ptr + n_vertices, sizeof(uint32_t), cudaMemcpyDeviceToHost, dev.stream),
                 "copy");
        GCU_TRY(dev.sync());
        GCU_TRY(b.row_list.allocate(dev, n_rows));
        GCU_TRY(row_graph.allocate(dev, n_rows));
        GCU_TRY(split_pos.allocate(dev, static_cast<uint64_t>(n_rows) + 1));
        GCU_TRY(b.lone.allocate(dev, n_vertices - n_rows));
        GCU_TRY(chunk_rows.allocate(dev, n_chunks));
        GCU_TRY(b.chunks.allocate(dev, n_chunks));
        GCU_TRY(b.chunk_lists.allocate(dev, 2 * n_chunks));
        GCU_TRY(b.delta.allocate(dev, n_chunks * kBatchChunk));
        GCU_CUDA(cudaMemsetAsync(b.lone_count.ptr, 0, 4ull * n_graphs, dev.stream), "memset");
        GCU_LAUNCH(dev, "batch_rows", batch_rows_kernel, small_grid(dev, n_vertices, 256), 256, 0, b.u.offsets.ptr,
                   b.large.ptr, n_graphs, n_vertices, pos.ptr, b.row_list.ptr, row_graph.ptr, b.lone.ptr,
                   b.lone_count.ptr, chunk_rows.ptr, split_pos.ptr);
        GCU_TRY(exclusive_scan_u32(dev, split_pos.ptr, split_pos.ptr, n_rows));
        GCU_CUDA(cudaMemcpyAsync(&n_split, split_pos.ptr + n_rows, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                 dev.stream),
                 "copy");
        if (n_chunks)
            GCU_LAUNCH(dev, "batch_chunks", batch_chunks_kernel, small_grid(dev, n_chunks, 8), 256, 0, b.u.offsets.ptr,
                       b.large.ptr, n_graphs, static_cast<uint32_t>(n_chunks), b.row_list.ptr, chunk_rows.ptr,
                       b.chunks.ptr, b.delta.ptr);
        GCU_TRY(dev.sync());
        GCU_TRY(b.split.allocate(dev, n_split));
        if (n_split)
            GCU_LAUNCH(dev, "batch_split_rows", batch_split_rows_kernel, small_grid(dev, n_rows, 256), 256, 0,
                       b.u.offsets.ptr, b.large.ptr, n_rows, b.row_list.ptr, row_graph.ptr, split_pos.ptr, b.split.ptr);
        b.rows = BatchRows{b.u.targets.ptr, b.large.ptr, b.row_list.ptr, b.chunks.ptr, b.delta.ptr, b.split.ptr, b.lone.ptr,
                           b.chunk_lists.ptr, n_graphs, n_rows, static_cast<uint32_t>(n_chunks), n_split,
                           static_cast<uint32_t>(n_vertices - n_rows)};
        GCU_TRY(dev.sync());
    }
    b.parted = true;
    return ok();
}

// Blocks of a pass kernel: all that are resident at once, fewer for large graphs
// too few to give every warp a turn.
template <class Kernel>
Error pass_grid(BatchImpl& b, Kernel kernel, unsigned* grid) {
    if (*grid) return ok();
    int per_sm = 0;
    GCU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBatchThreads, 0), "occupancy");
    const uint64_t most = static_cast<uint64_t>(b.dev->sm_count) * std::max(1, std::min(per_sm, kBatchCtasPerSm));
    const uint64_t want = std::max<uint64_t>(
        {1, ceil_div_u64(b.rows.n_chunks, kBatchThreads / 32),
         ceil_div_u64(static_cast<uint64_t>(b.rows.n_rows) + b.rows.n_lone, 4 * kBatchThreads)});
    *grid = static_cast<unsigned>(std::min(want, most));
    return ok();
}

// Blocks of a kernel over a class of the small graphs: as many as there are graphs,
// up to all that are resident.
template <class Kernel>
Error small_blocks(BatchImpl& b, Kernel kernel, int cls, unsigned* grid) {
    int per_sm = 0;
    GCU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSmallThreads[cls], 0), "occupancy");
    *grid = std::min<unsigned>(b.n_small[cls], static_cast<unsigned>(b.dev->sm_count) * std::max(1, per_sm));
    return ok();
}

BatchSmall small_graphs(const BatchImpl& b, int cls, uint32_t* next) {
    const BatchGraph* first = b.small.ptr;
    for (int c = 0; c < cls; ++c) first += b.n_small[c];
    return BatchSmall{b.u.offsets.ptr, b.u.targets.ptr, first, b.n_small[cls], next + cls};
}

template <int kClass>
Error launch_small_bfs(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    if (!b.n_small[kClass]) return ok();
    constexpr int kThreads = kSmallThreads[kClass];
    unsigned grid = 0;
    GCU_TRY(small_blocks(b, batch_small_bfs_kernel<kThreads>, kClass, &grid));
    const BatchSmallBfs a{small_graphs(b, kClass, b.next_small.ptr), b.sources.ptr, b.u.num_nodes, b.S, source_bits(b),
                          b.mask_a.ptr, b.mask_b.ptr, b.keep_dist ? b.dist.ptr : nullptr, b.reachable.ptr,
                          b.max_depth.ptr};
    GCU_LAUNCH(dev, "batch_small_bfs", batch_small_bfs_kernel<kThreads>, grid, kThreads, 0, a);
    return ok();
}

template <int kClass>
Error launch_small_ppr(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    if (!b.n_small[kClass]) return ok();
    constexpr int kThreads = kSmallThreads[kClass];
    unsigned grid = 0;
    GCU_TRY(small_blocks(b, batch_small_ppr_kernel<kThreads>, kClass, &grid));
    const BatchSmallPpr a{small_graphs(b, kClass, b.next_small.ptr + kSmallClasses), b.tele.ptr,
                          static_cast<double>(b.damping), static_cast<double>(b.tolerance), b.max_iterations,
                          b.contrib_a.ptr, b.contrib_b.ptr, b.ranks.ptr, b.iterations.ptr, b.converged.ptr};
    GCU_LAUNCH(dev, "batch_small_ppr", batch_small_ppr_kernel<kThreads>, grid, kThreads, 0, a);
    return ok();
}

Error launch_bfs(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    if (b.keep_dist)
        GCU_CUDA(cudaMemsetAsync(b.dist.ptr, 0xFF, sizeof(int32_t) * b.S * static_cast<size_t>(b.u.num_nodes),
                                 dev.stream),
                 "memset");
    if (b.rows.n_graphs) {
        GCU_TRY(pass_grid(b, batch_bfs_kernel, &b.bfs_grid));
        GCU_CUDA(cudaMemsetAsync(b.bfs_state.ptr, 0, sizeof(BatchRunState), dev.stream), "memset");
        const BatchBfs a{b.rows, b.sources.ptr, b.u.num_nodes, b.S, source_bits(b), b.mask_a.ptr, b.mask_b.ptr,
                         b.bfs_parts.ptr, b.keep_dist ? b.dist.ptr : nullptr, b.fresh.ptr, b.bfs_stop.ptr,
                         b.reachable.ptr, b.max_depth.ptr, b.bfs_state.ptr};
        GCU_LAUNCH_COOP(dev, "batch_bfs", batch_bfs_kernel, b.bfs_grid, kBatchThreads, 0, a);
    }
    GCU_CUDA(cudaMemsetAsync(b.next_small.ptr, 0, sizeof(uint32_t) * kSmallClasses, dev.stream), "memset");
    GCU_TRY(launch_small_bfs<0>(b));
    GCU_TRY(launch_small_bfs<1>(b));
    GCU_TRY(launch_small_bfs<2>(b));
    return ok();
}

Error launch_ppr(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    if (b.rows.n_graphs) {
        GCU_TRY(pass_grid(b, batch_ppr_kernel, &b.ppr_grid));
        GCU_CUDA(cudaMemsetAsync(b.ppr_state.ptr, 0, sizeof(BatchRunState), dev.stream), "memset");
        BatchPpr a{};
        a.rows = b.rows;
        a.lone_count = b.lone_count.ptr;
        a.tele = b.tele.ptr;
        a.lone_tele = b.lone_tele.ptr;
        a.K = b.K;
        while (a.log_lanes < 5 && (1u << a.log_lanes) < b.K) ++a.log_lanes;
        a.damp = static_cast<double>(b.damping);
        a.tolerance = static_cast<double>(b.tolerance);
        a.scale = kChangeUnits / a.tolerance;
        a.max_iterations = b.max_iterations;
        a.contrib_a = b.contrib_a.ptr;
        a.contrib_b = b.contrib_b.ptr;
        a.ranks = b.ranks.ptr;
        a.parts = b.ppr_parts.ptr;
        a.change = b.change.ptr;
        a.mass = b.mass.ptr;
        a.stop = b.ppr_stop.ptr;
        a.iterations = b.iterations.ptr;
        a.converged = b.converged.ptr;
        a.st = b.ppr_state.ptr;
        GCU_LAUNCH_COOP(dev, "batch_ppr", batch_ppr_kernel, b.ppr_grid, kBatchThreads, 0, a);
    }
    GCU_CUDA(cudaMemsetAsync(b.next_small.ptr + kSmallClasses, 0, sizeof(uint32_t) * kSmallClasses, dev.stream),
             "memset");
    GCU_TRY(launch_small_ppr<0>(b));
    GCU_TRY(launch_small_ppr<1>(b));
    GCU_TRY(launch_small_ppr<2>(b));
    return ok();
}

// A pass kernel's state, copied beside its results; check() after the
// synchronisation that ends the call.
struct RunCheck {
    BatchRunState state{};
    Error copy(BatchImpl& b, const DeviceBuffer<BatchRunState>& st) {
        if (b.rows.n_graphs)
            GCU_CUDA(cudaMemcpyAsync(&state, st.ptr, sizeof(state), cudaMemcpyDeviceToHost, b.dev->stream), "copy");
        return ok();
    }
    Error check(const char* what) const {
        return state.bar.failed ? kernel_error(std::string(what) + ": a block did not reach the grid barrier") : ok();
    }
};

Error launch_tc(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    GCU_TRY(batch_tc_launch(dev, *b.tc, b.tri_vertex.ptr, b.u.num_nodes));
    GCU_LAUNCH(dev, "batch_graph_sum", batch_graph_sum_kernel, small_grid(dev, b.G, 1), 256, 0, b.tri_vertex.ptr,
               b.d_vbase.ptr, b.G, b.tri_totals.ptr);
    return ok();
}

// Runs and times a pass kernel once on the whole batch (for batch_tuning).
template <class Launch>
Error timed_run(BatchImpl& b, Launch launch, std::string* json) {
    DeviceImpl& dev = *b.dev;
    cudaEvent_t e0, e1;
    GCU_CUDA(cudaEventCreate(&e0), "cudaEventCreate");
    GCU_CUDA(cudaEventCreate(&e1), "cudaEventCreate");
    cudaEventRecord(e0, dev.stream);
    Error err = launch(b);
    cudaEventRecord(e1, dev.stream);
    if (err.ok()) err = dev.sync();
    float ms = 0.f;
    if (err.ok()) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    const std::string threads = std::to_string(kBatchThreads);
    *json = "{\"" + threads + "\": " + std::to_string(ms) + ", \"chosen\": " + threads + "}";
    return err;
}

}  // namespace

// The generated corpus: graph i is R-MAT (scale U{8..16}, edge factor
// U{8..32}, a, b, c = 0.57, 0.19, 0.19) or Watts-Strogatz (n U{256..65536},
// k = 10, p = 0.1) with equal odds, every draw from SplitMix64 of (seed, i).
Error batch_generate(DeviceImpl& dev, std::shared_ptr<DeviceImpl> owner, uint32_t num_graphs, uint64_t seed,
                     BatchImpl** out) {
    auto b = std::make_unique<BatchImpl>();
    b->dev = owner;
    b->u.dev = owner;
    b->G = num_graphs;
    std::vector<GeneratorSpec> specs(num_graphs);
    for (uint32_t i = 0; i < num_graphs; ++i) {
        const uint64_t r = mix64(mix64(seed + 0x9E3779B97F4A7C15ull) + i);
        GeneratorSpec& s = specs[i];
        s.seed = mix64(r ^ 0xD1B54A32D192ED03ull);
        if ((r & 1) == 0) {
            s.kind = GeneratorSpec::kRmat;
            s.scale = 8 + static_cast<uint32_t>((r >> 8) % 9);
            s.edge_factor = 8 + static_cast<uint32_t>((r >> 16) % 25);
            s.a = 0.57;
            s.b = 0.19;
            s.c = 0.19;
        } else {
            s.kind = GeneratorSpec::kWattsStrogatz;
            s.n = 256 + static_cast<uint32_t>((r >> 8) % (65536 - 256 + 1));
            s.k = 10;
            s.p = 0.1;
        }
    }
    GCU_TRY(generate_union(dev, specs, &b->vbase, b->u));
    GCU_TRY(finish_layout(*b));
    *out = b.release();
    return ok();
}

Error batch_from_csr(DeviceImpl& dev, std::shared_ptr<DeviceImpl> owner, const uint32_t* vbase, size_t num_graphs,
                     const uint32_t* offsets, size_t n_offsets, const uint32_t* targets, size_t n_targets,
                     BatchImpl** out) {
    if (n_offsets == 0) return invalid_csr("offsets must have num_nodes + 1 entries, got an empty array");
    if (vbase[0] != 0 || vbase[num_graphs] != n_offsets - 1)
        return kernel_error("vertex_base must start at 0 and end at num_nodes (" + std::to_string(n_offsets - 1) +
                            ")");
    for (size_t i = 0; i < num_graphs; ++i)
        if (vbase[i + 1] < vbase[i]) return kernel_error("vertex_base must be non-decreasing");
    if (offsets[0] != 0) return invalid_csr("offsets[0] must be 0, got " + std::to_string(offsets[0]));
    if (static_cast<size_t>(offsets[n_offsets - 1]) != n_targets)
        return invalid_csr("offsets[" + std::to_string(n_offsets - 1) + "] is " +
                           std::to_string(offsets[n_offsets - 1]) + " but targets has " + std::to_string(n_targets) +
                           " entries");
    auto b = std::make_unique<BatchImpl>();
    b->dev = owner;
    b->u.dev = owner;
    b->G = static_cast<uint32_t>(num_graphs);
    b->vbase.assign(vbase, vbase + num_graphs + 1);
    GraphImpl& u = b->u;
    u.num_nodes = static_cast<uint32_t>(n_offsets - 1);
    u.num_edges = static_cast<uint32_t>(n_targets);
    GCU_TRY(u.offsets.allocate(dev, n_offsets));
    GCU_TRY(u.targets.allocate(dev, n_targets));
    GCU_TRY(copy_to_device(dev, u.offsets.ptr, offsets, 4 * n_offsets, dev.stream));
    if (n_targets)
        GCU_TRY(copy_to_device(dev, u.targets.ptr, targets, 4 * n_targets, dev.stream));
    uint32_t bad = UINT32_MAX;
    GCU_TRY(validate_csr_device(dev, u.offsets.ptr, u.targets.ptr, u.num_nodes, u.num_edges, &bad));
    if (bad != UINT32_MAX) {
        const uint32_t start = offsets[bad], end = offsets[bad + 1];
        const size_t lo = std::min<size_t>(start, n_targets), hi = std::min<size_t>(std::max(start, end), n_targets);
        return invalid_csr(describe_node_violation(bad, start, end, targets + lo, hi - lo, u.num_nodes));
    }
    GCU_TRY(finish_layout(*b));
    DeviceBuffer<unsigned long long> first;
    GCU_TRY(first.allocate(dev, 1));
    GCU_CUDA(cudaMemsetAsync(first.ptr, 0xFF, sizeof(unsigned long long), dev.stream), "memset");
    GCU_LAUNCH(dev, "batch_check", batch_check_kernel, small_grid(dev, b->G, 1), 256, 0, u.offsets.ptr, u.targets.ptr,
               b->d_vbase.ptr, b->G, first.ptr);
    unsigned long long j = 0;
    GCU_CUDA(cudaMemcpyAsync(&j, first.ptr, sizeof(j), cudaMemcpyDeviceToHost, dev.stream), "copy");
    GCU_TRY(dev.sync());
    if (j != ~0ull) {
        const uint32_t row = static_cast<uint32_t>(std::upper_bound(offsets, offsets + n_offsets, j) - offsets - 1);
        return kernel_error("batch: edge (" + std::to_string(row) + ", " + std::to_string(targets[j]) +
                            ") leaves its graph");
    }
    *out = b.release();
    return ok();
}

Error batch_member(BatchImpl& b, uint32_t index, GraphImpl& g) {
    DeviceImpl& dev = *b.dev;
    if (index >= b.G) return kernel_error("graph index " + std::to_string(index) + " out of range (batch of " +
                                          std::to_string(b.G) + ")");
    const uint32_t vb = b.vbase[index], n = b.vbase[index + 1] - vb;
    const uint32_t eb = b.ebase[index], m = b.ebase[index + 1] - eb;
    g.num_nodes = n;
    g.num_edges = m;
    GCU_TRY(g.offsets.allocate(dev, static_cast<uint64_t>(n) + 1));
    GCU_TRY(g.targets.allocate(dev, m));
    GCU_LAUNCH(dev, "batch_extract", batch_extract_kernel, small_grid(dev, std::max<uint64_t>(n + 1, m), 256), 256, 0,
               b.u.offsets.ptr, b.u.targets.ptr, vb, n, eb, m, g.offsets.ptr, g.targets.ptr);
    g.symmetric = b.u.symmetric;
    return dev.sync();
}

// A captured graph holds the device pointers and the per-batch parameters
// (S, K, damping, ...) by value: setting new sources or seeds reallocates the
// buffers it reads, so the capture is dropped, and gcu_batch_replay refuses
// to run until the caller captures again.
static void drop_capture(BatchImpl& b) {
    if (b.exec) {
        cudaGraphExecDestroy(b.exec);
        b.exec = nullptr;
    }
    if (b.graph) {
        cudaGraphDestroy(b.graph);
        b.graph = nullptr;
    }
}

Error batch_set_bfs(BatchImpl& b, const uint32_t* sources, uint32_t S, bool keep_distances) {
    DeviceImpl& dev = *b.dev;
    if (S == 0 || S > kMaxBatchSources) return kernel_error("sources per graph must be in 1..=32");
    for (uint32_t g = 0; g < b.G; ++g) {
        const uint32_t n = b.vbase[g + 1] - b.vbase[g];
        for (uint32_t k = 0; k < S; ++k)
            if (sources[static_cast<uint64_t>(g) * S + k] >= n)
                return kernel_error("source node " + std::to_string(sources[static_cast<uint64_t>(g) * S + k]) +
                                    " of graph " + std::to_string(g) + " out of range (num_nodes = " +
                                    std::to_string(n) + ")");
    }
    GCU_TRY(dev.sync());  // a replay in flight may still read the old buffers
    drop_capture(b);
    GCU_TRY(part_graphs(b));
    const uint64_t V = b.u.num_nodes;
    b.S = S;
    b.keep_dist = keep_distances;
    GCU_TRY(b.sources.allocate(dev, static_cast<uint64_t>(b.G) * S));
    GCU_CUDA(cudaMemcpyAsync(b.sources.ptr, sources, 4ull * b.G * S, cudaMemcpyHostToDevice, dev.stream), "copy");
    GCU_TRY(b.bfs_parts.allocate(dev, 2ull * b.rows.n_chunks));
    GCU_TRY(b.fresh.allocate(dev, 3ull * b.rows.n_graphs));
    GCU_TRY(b.bfs_stop.allocate(dev, b.rows.n_graphs));
    GCU_TRY(b.mask_a.allocate(dev, V));
    GCU_TRY(b.mask_b.allocate(dev, V));
    GCU_TRY(b.reachable.allocate(dev, static_cast<uint64_t>(b.G) * S));
    GCU_TRY(b.max_depth.allocate(dev, static_cast<uint64_t>(b.G) * S));
    if (keep_distances) GCU_TRY(b.dist.allocate(dev, V * S));
    b.bfs_timed = false;
    return dev.sync();
}

Error batch_set_ppr(BatchImpl& b, const uint32_t* seeds, uint32_t K, float damping, uint32_t max_iterations,
                    float tolerance) {
    DeviceImpl& dev = *b.dev;
    if (K == 0) return kernel_error("personalized PageRank needs at least one seed");
    for (uint32_t g = 0; g < b.G; ++g) {
        const uint32_t n = b.vbase[g + 1] - b.vbase[g];
        for (uint32_t k = 0; k < K; ++k)
            if (seeds[static_cast<uint64_t>(g) * K + k] >= n)
                return kernel_error("seed node " + std::to_string(seeds[static_cast<uint64_t>(g) * K + k]) +
                                    " of graph " + std::to_string(g) + " out of range (num_nodes = " +
                                    std::to_string(n) + ")");
    }
    GCU_TRY(dev.sync());  // a replay in flight may still read the old buffers
    drop_capture(b);
    GCU_TRY(part_graphs(b));
    const uint64_t V = b.u.num_nodes;
    b.K = K;
    b.damping = damping;
    b.max_iterations = max_iterations;
    b.tolerance = tolerance;
    GCU_TRY(b.seeds.allocate(dev, static_cast<uint64_t>(b.G) * K));
    GCU_CUDA(cudaMemcpyAsync(b.seeds.ptr, seeds, 4ull * b.G * K, cudaMemcpyHostToDevice, dev.stream), "copy");
    GCU_TRY(b.tele.allocate(dev, V));
    GCU_TRY(b.ppr_parts.allocate(dev, 2ull * b.rows.n_chunks));
    GCU_TRY(b.change.allocate(dev, 3ull * b.rows.n_graphs));
    GCU_TRY(b.mass.allocate(dev, 2ull * b.rows.n_graphs));
    GCU_TRY(b.lone_tele.allocate(dev, static_cast<uint64_t>(b.G) * K));
    GCU_TRY(b.ppr_stop.allocate(dev, b.rows.n_graphs));
    GCU_TRY(b.contrib_a.allocate(dev, V));
    GCU_TRY(b.contrib_b.allocate(dev, V));
    GCU_TRY(b.ranks.allocate(dev, V));
    GCU_TRY(b.iterations.allocate(dev, std::max<uint32_t>(b.G, 1)));
    GCU_TRY(b.converged.allocate(dev, std::max<uint32_t>(b.G, 1)));
    GCU_CUDA(cudaMemsetAsync(b.tele.ptr, 0, 4 * std::max<uint64_t>(V, 1), dev.stream), "memset");
    GCU_LAUNCH(dev, "batch_tele", batch_tele_kernel, small_grid(dev, static_cast<uint64_t>(b.G) * K, 256), 256, 0,
               b.seeds.ptr, b.d_vbase.ptr, b.G, K, b.tele.ptr);
    // Each graph's seeds once, in order, then their teleports where they have no entries.
    if (K > 1) {
        std::vector<uint32_t> once(seeds, seeds + static_cast<uint64_t>(b.G) * K);
        for (auto first = once.begin(); first != once.end(); first += K) {
            if (!std::is_sorted(first, first + K)) std::sort(first, first + K);
            std::fill(std::unique(first, first + K), first + K, kNoSeed);
        }
        GCU_CUDA(cudaMemcpyAsync(b.seeds.ptr, once.data(), 4ull * b.G * K, cudaMemcpyHostToDevice, dev.stream), "copy");
    }
    GCU_LAUNCH(dev, "batch_lone_tele", batch_lone_tele_kernel, small_grid(dev, static_cast<uint64_t>(b.G) * K, 256), 256,
               0, b.seeds.ptr, b.d_vbase.ptr, b.u.offsets.ptr, b.tele.ptr, b.G, K, b.lone_tele.ptr);
    b.ppr_timed = false;
    return dev.sync();
}

Error batch_ensure_tc(BatchImpl& b) {
    if (b.tc) return ok();
    DeviceImpl& dev = *b.dev;
    GCU_TRY(b.tri_vertex.allocate(dev, std::max<uint32_t>(b.u.num_nodes, 1)));
    GCU_TRY(b.tri_totals.allocate(dev, std::max<uint32_t>(b.G, 1)));
    return batch_tc_plan(b.u, &b.tc, &b.tc_tuning);
}

Error batch_run_tc(BatchImpl& b, uint64_t* totals) {
    GCU_TRY(batch_ensure_tc(b));
    GCU_TRY(launch_tc(b));
    GCU_CUDA(cudaMemcpyAsync(totals, b.tri_totals.ptr, 8ull * b.G, cudaMemcpyDeviceToHost, b.dev->stream), "copy");
    return b.dev->sync();
}

Error batch_run_bfs(BatchImpl& b) {
    if (!b.S) return kernel_error("batch BFS sources are not set");
    if (b.bfs_timed) {
        GCU_TRY(launch_bfs(b));
    } else {
        GCU_TRY(timed_run(b, launch_bfs, &b.bfs_tuning));
        b.bfs_timed = true;
    }
    return b.dev->sync();
}

Error batch_run_ppr(BatchImpl& b) {
    if (!b.K) return kernel_error("batch PageRank seeds are not set");
    if (b.ppr_timed) {
        GCU_TRY(launch_ppr(b));
    } else {
        GCU_TRY(timed_run(b, launch_ppr, &b.ppr_tuning));
        b.ppr_timed = true;
    }
    return b.dev->sync();
}

Error batch_read_bfs(BatchImpl& b, int32_t* distances, uint32_t* reachable, int32_t* max_depth) {
    DeviceImpl& dev = *b.dev;
    const uint64_t gs = static_cast<uint64_t>(b.G) * b.S;
    RunCheck run;
    GCU_TRY(run.copy(b, b.bfs_state));
    if (distances && b.keep_dist) GCU_TRY(copy_to_host(dev, distances, b.dist.ptr, 4ull * b.S * b.u.num_nodes));
    if (reachable) GCU_CUDA(cudaMemcpyAsync(reachable, b.reachable.ptr, 4 * gs, cudaMemcpyDeviceToHost, dev.stream), "copy");
    if (max_depth) GCU_CUDA(cudaMemcpyAsync(max_depth, b.max_depth.ptr, 4 * gs, cudaMemcpyDeviceToHost, dev.stream), "copy");
    GCU_TRY(dev.sync());
    return run.check("batch BFS");
}

Error batch_read_ppr(BatchImpl& b, float* ranks, uint32_t* iterations, uint8_t* converged) {
    DeviceImpl& dev = *b.dev;
    RunCheck run;
    GCU_TRY(run.copy(b, b.ppr_state));
    if (ranks) GCU_TRY(copy_to_host(dev, ranks, b.ranks.ptr, 4ull * b.u.num_nodes));
    if (iterations)
        GCU_CUDA(cudaMemcpyAsync(iterations, b.iterations.ptr, 4ull * b.G, cudaMemcpyDeviceToHost, dev.stream), "copy");
    if (converged)
        GCU_CUDA(cudaMemcpyAsync(converged, b.converged.ptr, b.G, cudaMemcpyDeviceToHost, dev.stream), "copy");
    GCU_TRY(dev.sync());
    return run.check("batch PageRank");
}

// Captures triangle counts, BFS and PageRank of the whole batch into one CUDA
// graph (planned and run once first: nothing in the capture allocates or syncs).
Error batch_capture(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    if (!b.S || !b.K) return kernel_error("set the batch BFS sources and PageRank seeds before capturing");
    GCU_TRY(batch_ensure_tc(b));
    if (!b.bfs_timed) GCU_TRY(batch_run_bfs(b));
    if (!b.ppr_timed) GCU_TRY(batch_run_ppr(b));
    drop_capture(b);
    const bool timing = dev.kernel_timing;
    dev.kernel_timing = false;  // no event bookkeeping inside the capture
    GCU_CUDA(cudaStreamBeginCapture(dev.stream, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
    Error e = launch_tc(b);
    if (e.ok()) e = launch_bfs(b);
    if (e.ok()) e = launch_ppr(b);
    cudaGraph_t graph = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(dev.stream, &graph);
    dev.kernel_timing = timing;
    if (!e.ok()) {
        if (graph) cudaGraphDestroy(graph);
        return e;
    }
    if (ce != cudaSuccess) return driver_error(ce, "cudaStreamEndCapture");
    b.graph = graph;
    GCU_CUDA(cudaGraphInstantiate(&b.exec, b.graph, 0), "cudaGraphInstantiate");
    return ok();
}

Error batch_replay(BatchImpl& b) {
    if (!b.exec) return kernel_error("batch has no captured graph (call gcu_batch_capture first)");
    b.dev->launches.fetch_add(1, std::memory_order_relaxed);
    GCU_CUDA(cudaGraphLaunch(b.exec, b.dev->stream), "cudaGraphLaunch");
    return ok();
}

uint32_t batch_num_graphs(const BatchImpl& b) { return b.G; }
GraphImpl& batch_union(BatchImpl& b) { return b.u; }
const std::vector<uint32_t>& batch_vertex_base(const BatchImpl& b) { return b.vbase; }

Error batch_read_tc(BatchImpl& b, uint64_t* totals) {
    if (!b.tc) return kernel_error("batch triangle counts have not run");
    GCU_CUDA(cudaMemcpyAsync(totals, b.tri_totals.ptr, 8ull * b.G, cudaMemcpyDeviceToHost, b.dev->stream), "copy");
    return b.dev->sync();
}

std::string batch_tuning(const BatchImpl& b) {
    return "{\"triangle_buckets\": " + (b.tc_tuning.empty() ? std::string("null") : b.tc_tuning) +
           ", \"bfs_threads\": " + (b.bfs_tuning.empty() ? std::string("null") : b.bfs_tuning) +
           ", \"ppr_threads\": " + (b.ppr_tuning.empty() ? std::string("null") : b.ppr_tuning) + "}";
}

}  // namespace gcu

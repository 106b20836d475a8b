// Batched form: many uneven graphs packed into one CSR and processed by
// persistent kernels, replayed as one captured CUDA graph.
//
// Layout: graph i owns the vertices [vbase[i], vbase[i + 1]) of a union CSR
// whose targets are union ids (no edge leaves its graph), so the union is a
// plain symmetric CSR and graph i's entries are [offsets[vbase[i]],
// offsets[vbase[i + 1]]).
//
//  * Triangles: word lists of the union, counted per owner (tri_words.cu), or,
//    with a learned schedule installed, one degree-oriented DAG of the union and
//    its out-degree buckets, the schedule's variant per bucket; a block per graph
//    sums its vertices.
//  * BFS and PageRank run over the union as a whole, one cooperative launch
//    each: every level or iteration is one pass over the entries of all graphs
//    that are still at work, and the blocks meet at a grid barrier. The entries
//    are read as a stream of 256-entry chunks (8 consecutive entries per lane,
//    a byte per entry says which row it belongs to), so a pass is spread evenly
//    over the GPU whatever the sizes of the graphs; a graph has no CTA of its
//    own to wait for. Rows that cross chunks leave parts that are joined after
//    the pass.
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
constexpr uint32_t kNoGraph = 0xFFFFFFFFu;

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

// The union's rows with entries, packed ("rows" below are indices into this
// list), and its vertices without.
struct BatchRows {
    const uint32_t* targets;
    const uint32_t* row_vertex;  // union vertex of each row
    const uint32_t* row_graph;
    const uint32_t* row_start;   // first entry of each row; [n_rows] = E
    const uint32_t* chunk_row;   // row of each chunk's first entry
    const uint8_t* delta;        // per entry: its row minus its chunk's first row
    const uint4* split;          // (row, first chunk, last chunk, 0) of the rows that cross chunks
    const uint32_t* lone;        // vertices without entries
    const uint32_t* lone_graph;
    uint32_t E, n_rows, n_chunks, n_split, n_lone;
};

struct BatchRunState {
    GridBarrier bar;
    uint32_t active[3];  // graphs at work in this pass, rotating
};

__global__ void batch_row_flags_kernel(const uint32_t* __restrict__ offsets, uint32_t V, uint32_t* __restrict__ flag) {
    for (uint64_t v = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
         v += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        flag[v] = offsets[v + 1] > offsets[v] ? 1u : 0u;
}

__global__ void batch_rows_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ pos,
                                  const uint32_t* __restrict__ vbase, uint32_t G, uint32_t V, uint32_t E,
                                  uint32_t* __restrict__ row_vertex, uint32_t* __restrict__ row_graph,
                                  uint32_t* __restrict__ row_start, uint32_t* __restrict__ lone,
                                  uint32_t* __restrict__ lone_graph, uint32_t* __restrict__ lone_count) {
    for (uint64_t v = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v <= V;
         v += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        if (v == V) {
            row_start[pos[V]] = E;
            continue;
        }
        // The last graph that begins at or before v (empty graphs share a base with their successor).
        uint32_t lo = 0, hi = G;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (vbase[mid] <= v) lo = mid;
            else hi = mid;
        }
        const uint32_t r = pos[v], i = static_cast<uint32_t>(v) - r;
        if (pos[v + 1] > r) {
            row_vertex[r] = static_cast<uint32_t>(v);
            row_graph[r] = lo;
            row_start[r] = offsets[v];
        } else {
            lone[i] = static_cast<uint32_t>(v);
            lone_graph[i] = lo;
            atomicAdd(lone_count + lo, 1u);
        }
    }
}

__global__ void batch_chunk_rows_kernel(const uint32_t* __restrict__ row_start, uint32_t n_rows,
                                        uint32_t* __restrict__ chunk_row, uint32_t* __restrict__ split_flag) {
    for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n_rows;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t s = row_start[r], e = row_start[r + 1];
        const uint64_t c_first = s / kBatchChunk, c_last = (e - 1) / kBatchChunk;
        for (uint64_t c = (s + kBatchChunk - 1) / kBatchChunk; c <= c_last; ++c) chunk_row[c] = static_cast<uint32_t>(r);
        split_flag[r] = c_first != c_last ? 1u : 0u;
    }
}

__global__ void batch_split_rows_kernel(const uint32_t* __restrict__ row_start, uint32_t n_rows,
                                        const uint32_t* __restrict__ pos, uint4* __restrict__ split) {
    for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n_rows;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        if (pos[r + 1] > pos[r])
            split[pos[r]] = make_uint4(static_cast<uint32_t>(r), row_start[r] / kBatchChunk,
                                       (row_start[r + 1] - 1) / kBatchChunk, 0u);
}

__global__ void __launch_bounds__(256) batch_delta_kernel(const uint32_t* __restrict__ row_start, uint32_t n_rows,
                                                          uint32_t E, const uint32_t* __restrict__ chunk_row,
                                                          uint8_t* __restrict__ delta) {
    for_each_entry<256, 4>(row_start, n_rows, E, [&](uint32_t j, uint32_t r) {
        delta[j] = static_cast<uint8_t>(r - chunk_row[j / kBatchChunk]);
    });
}

// One pass: chunk after chunk, a warp each (kBatchRun consecutive chunks per
// turn), 8 consecutive entries per lane. op gives
//   begin(g0, g1)      whether a graph in [g0, g1] is at work (else the chunk is skipped)
//   want(row)          whether the row's entries have to be gathered
//   gather(target), add(x, y), zero()
//   load(row), more(in)  what finish needs besides the result: loads, and those
//                      that depend on them
//   finish(row, x, in) the row's result
//   part(i, x)         part i of a row that crosses chunks: 2c for the end of a row
//                      begun before chunk c, 2c + 1 for a row that goes on after it
//   flush()            after every turn (all lanes)
// Runs of equal rows are joined per lane, then across lanes by a segmented
// scan; the lane where a row ends puts its result into s_row (kBatchChunk of the
// warp's own), from where consecutive lanes finish consecutive rows. The first 32
// rows' inputs are loaded beside the gathers: loads that follow them wait in the
// queue behind them.
template <class Op>
__device__ __forceinline__ void batch_pass(const BatchRows& R, Op& op, typename Op::T* s_row) {
    using T = typename Op::T;
    const unsigned lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    for (uint64_t c0 = static_cast<uint64_t>(warp) * kBatchRun; c0 < R.n_chunks;
         c0 += static_cast<uint64_t>(warps) * kBatchRun) {
        const uint32_t c1 = static_cast<uint32_t>(min_u64(c0 + kBatchRun, R.n_chunks));
        for (uint32_t c = static_cast<uint32_t>(c0); c < c1; ++c) {
            const uint64_t e0 = static_cast<uint64_t>(c) * kBatchChunk;
            const uint64_t eb = e0 + 8 * lane;
            const uint32_t rbase = __ldg(R.chunk_row + c);
            const uint2 dl = ld_stream2(reinterpret_cast<const uint2*>(R.delta + eb));
            const bool any = eb < R.E;
            uint32_t row[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                row[i] = eb + i < R.E ? rbase + (((i < 4 ? dl.x : dl.y) >> (8 * (i & 3))) & 0xFFu) : kNoGraph;
            // The last row: of the last entry (only the last chunk can end early).
            const uint64_t last = min_u64(e0 + kBatchChunk, R.E) - 1 - e0;
            const uint32_t mine_last = rbase + ((last & 4 ? dl.y : dl.x) >> (8 * (last & 3)) & 0xFFu);
            const uint32_t rlast = __shfl_sync(kFullMask, mine_last, static_cast<int>(last >> 3));
            if (!op.begin(__ldg(R.row_graph + rbase), __ldg(R.row_graph + rlast))) continue;
            const bool first_split = __ldg(R.row_start + rbase) < e0;
            const bool last_split = __ldg(R.row_start + rlast + 1) > e0 + kBatchChunk;
            bool want[8];
            bool some = false;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (!Op::kSkips) want[i] = row[i] != kNoGraph;
                else if (i > 0 && row[i] == row[i - 1]) want[i] = want[i - 1];
                else want[i] = row[i] != kNoGraph && op.want(row[i]);
                some = some || want[i];
            }
            uint32_t t[8] = {};
            if (Op::kSkips ? some : any) ld_stream8(R.targets + eb, t);
            const uint32_t n_rows = rlast - rbase + 1;
            auto in = op.load(rbase + min(lane, n_rows - 1));
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
                        s_row[row[i] - rbase] = acc;
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
            if (multi && rf != kNoGraph) s_row[rf - rbase] = carry_in ? Op::add(head, carry) : head;
            const bool continues = lane < 31 && next_first == rl;
            if (!continues && rl != kNoGraph) s_row[rl - rbase] = S;  // the last run ends at this lane's end
            __syncwarp();
            for (uint32_t r = lane; r < n_rows; r += 32) {
                if (r >= 32) {
                    in = op.load(rbase + r);
                    op.more(in);
                }
                const T x = s_row[r];
                if (r == n_rows - 1 && last_split) op.part(2 * static_cast<uint64_t>(c) + 1, x);
                else if (r == 0 && first_split) op.part(2 * static_cast<uint64_t>(c), x);
                else op.finish(rbase + r, x, in);
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
        if (i < R.n_split) {
            const uint4 s = R.split[i];
            const uint32_t g = __ldg(R.row_graph + s.x);
            if (op.begin(g, g)) {
                T x = op.parts(2 * static_cast<uint64_t>(s.y) + 1);
                for (uint32_t c = s.y + 1; c < s.z; ++c) x = Op::add(x, op.parts(2 * static_cast<uint64_t>(c) + 1));
                x = Op::add(x, op.parts(2 * static_cast<uint64_t>(s.z)));
                auto in = op.load(s.x);
                op.more(in);
                op.finish(s.x, x, in);
            }
        }
        op.flush();
    }
}

// ---------------------------------------------------------------- multi-source BFS

struct BatchBfs {
    BatchRows rows;
    const uint32_t* offsets;
    const uint32_t* vbase;
    const uint32_t* sources;
    uint32_t G, V, S, full;
    uint32_t *mask_a, *mask_b;
    uint32_t* parts;
    int32_t* dist;  // NULL: no distances
    uint32_t* fresh;      // [3][G]: sources that reached something new, rotating by level
    uint32_t* stop;       // [G]: the level a graph stopped before
    uint32_t* reachable;
    int32_t* max_depth;
    BatchRunState* st;
};

struct BfsOp {
    using T = uint32_t;
    static constexpr bool kSkips = true;
    const BatchBfs& a;
    const uint32_t* in;
    uint32_t* out;
    const uint32_t* prev_fresh;  // [G], the level before (NULL at level 0)
    uint32_t* fresh;
    uint32_t level;
    uint32_t my_graph = kNoGraph, my_fresh = 0;

    static __device__ __forceinline__ T zero() { return 0u; }
    static __device__ __forceinline__ T add(T x, T y) { return x | y; }
    // A graph works on while the level before found something new.
    __device__ __forceinline__ bool works(uint32_t g) const {
        return a.stop[g] > level && (prev_fresh == nullptr || prev_fresh[g] != 0);
    }
    __device__ __forceinline__ bool begin(uint32_t g0, uint32_t g1) const {
        for (uint32_t g = g0; g <= g1; ++g)
            if (works(g)) return true;
        return false;
    }
    __device__ __forceinline__ bool want(uint32_t r) const { return in[__ldg(a.rows.row_vertex + r)] != a.full; }
    __device__ __forceinline__ T gather(bool p, uint32_t t) const { return ld_if(p, in + t, 0u); }
    __device__ __forceinline__ void part(uint64_t i, T x) { a.parts[i] = x; }
    __device__ __forceinline__ T parts(uint64_t i) const { return a.parts[i]; }
    struct In {
        uint32_t v, g, old;
    };
    __device__ __forceinline__ In load(uint32_t r) const {
        return In{__ldg(a.rows.row_vertex + r), __ldg(a.rows.row_graph + r), 0u};
    }
    __device__ __forceinline__ void more(In& x) const { x.old = ld_if(true, in + x.v, 0u); }
    __device__ __forceinline__ void finish(uint32_t, T m, const In& x) {
        const uint32_t v = x.v, old = x.old, now = (m & ~old);
        out[v] = old | m;
        if (!now) return;
        if (a.dist)
            for (uint32_t bits = now; bits; bits &= bits - 1)
                a.dist[static_cast<uint64_t>(__ffs(bits) - 1) * a.V + v] = static_cast<int32_t>(level) + 1;
        const uint32_t g = x.g;
        if (g != my_graph) {
            if (my_fresh) atomicOr(fresh + my_graph, my_fresh);
            my_graph = g;
            my_fresh = 0;
        }
        my_fresh |= now;
    }
    __device__ __forceinline__ void flush() {
        const unsigned has = __ballot_sync(kFullMask, my_fresh != 0);
        if (has) {
            const uint32_t g = __shfl_sync(kFullMask, my_graph, __ffs(has) - 1);
            const uint32_t bits = __reduce_or_sync(kFullMask, my_graph == g ? my_fresh : 0u);
            if (lane_id() == static_cast<unsigned>(__ffs(has) - 1)) atomicOr(fresh + g, bits);
            if (my_fresh && my_graph != g) atomicOr(fresh + my_graph, my_fresh);
        }
        my_graph = kNoGraph;
        my_fresh = 0;
    }
};

__global__ void __launch_bounds__(kBatchThreads, kBatchCtasPerSm) batch_bfs_kernel(const BatchBfs a) {
    __shared__ uint32_t s_active;
    __shared__ uint32_t s_count[kMaxBatchSources];
    __shared__ uint32_t s_rows[kBatchThreads / 32][kBatchChunk];
    const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t nthreads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    unsigned barriers = 0;
    for (uint64_t v = tid; v < a.V; v += nthreads) {
        a.mask_a[v] = 0;
        a.mask_b[v] = 0;
    }
    for (uint64_t g = tid; g < a.G; g += nthreads) {
        for (int q = 0; q < 3; ++q) a.fresh[static_cast<uint64_t>(q) * a.G + g] = 0;
        a.stop[g] = a.vbase[g + 1] > a.vbase[g] ? 0xFFFFFFFFu : 0u;
    }
    for (uint64_t i = tid; i < static_cast<uint64_t>(a.G) * a.S; i += nthreads) {
        a.reachable[i] = 0;
        a.max_depth[i] = 0;
    }
    if (!grid_barrier(&a.st->bar, barriers)) return;
    for (uint64_t i = tid; i < static_cast<uint64_t>(a.G) * a.S; i += nthreads) {
        const uint32_t g = static_cast<uint32_t>(i / a.S), k = static_cast<uint32_t>(i % a.S);
        const uint32_t v = a.vbase[g] + a.sources[i];
        // Both arrays: a vertex without entries is never written again.
        atomicOr(a.mask_a + v, 1u << k);
        atomicOr(a.mask_b + v, 1u << k);
        if (a.dist) a.dist[static_cast<uint64_t>(k) * a.V + v] = 0;
    }
    if (!grid_barrier(&a.st->bar, barriers)) return;
    // Each level labels something in some graph, or is the last.
    for (uint32_t level = 0;; ++level) {
        BfsOp op{a, (level & 1) ? a.mask_b : a.mask_a, (level & 1) ? a.mask_a : a.mask_b,
                 level ? a.fresh + static_cast<uint64_t>((level + 2) % 3) * a.G : nullptr,
                 a.fresh + static_cast<uint64_t>(level % 3) * a.G, level};
        for (uint64_t g = tid; g < a.G; g += nthreads) {
            a.fresh[static_cast<uint64_t>((level + 1) % 3) * a.G + g] = 0;  // last read a level ago
            if (a.stop[g] <= level) continue;
            if (level) {
                uint32_t bits = op.prev_fresh[g];
                if (!bits) {
                    a.stop[g] = level;
                    continue;
                }
                for (; bits; bits &= bits - 1)
                    a.max_depth[g * static_cast<uint64_t>(a.S) + __ffs(bits) - 1] = static_cast<int32_t>(level);
            }
            atomicAdd(a.st->active + level % 3, 1u);
        }
        if (tid == 0) a.st->active[(level + 1) % 3] = 0;
        batch_pass(a.rows, op, s_rows[threadIdx.x >> 5]);
        if (!grid_barrier(&a.st->bar, gridDim.x, barriers, [&] { s_active = __ldcg(a.st->active + level % 3); })) return;
        if (s_active == 0) break;
        batch_split_pass(a.rows, op);
        if (!grid_barrier(&a.st->bar, barriers)) return;
    }
    // Reached vertices per source: lane k of every warp counts bit k of its
    // graph's vertices. A graph that has stopped has the same masks in both arrays.
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    for (uint32_t g = blockIdx.x; g < a.G; g += gridDim.x) {
        if (threadIdx.x < kMaxBatchSources) s_count[threadIdx.x] = 0;
        __syncthreads();
        uint32_t cnt = 0;
        const uint32_t ve = a.vbase[g + 1];
        for (uint64_t base = static_cast<uint64_t>(a.vbase[g]) + warp * 32; base < ve; base += kBatchThreads) {
            const uint64_t v = base + lane;
            const uint32_t vis = v < ve ? a.mask_a[v] : 0u;
            for (uint32_t k = 0; k < a.S; ++k) {
                const unsigned b = __ballot_sync(kFullMask, (vis >> k) & 1u);
                if (lane == k) cnt += __popc(b);
            }
        }
        if (lane < a.S && cnt) atomicAdd(&s_count[lane], cnt);
        __syncthreads();
        if (threadIdx.x < a.S) a.reachable[static_cast<uint64_t>(g) * a.S + threadIdx.x] = s_count[threadIdx.x];
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

struct BatchPpr {
    BatchRows rows;
    const uint32_t* vbase;
    const uint32_t* lone_count;  // [G]
    const float* tele;
    const float* lone_tele;      // [G][K] of the seeds without entries (each once), 0 for the others
    uint32_t G, V, K, log_lanes; // 2^log_lanes lanes sum a graph's dangling mass
    double damp, tolerance, scale;
    uint32_t max_iterations;
    float *contrib_a, *contrib_b;
    float* ranks;
    double* parts;
    ChangeSum* change;           // [3][G], rotating by iteration
    double* mass;                // [2][G]: dangling mass, alternating
    uint32_t* stop;              // [G]: iterations a graph has run when it stopped
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
    const ChangeSum* prev_change;  // [G], the iteration before
    const double* mass;            // [G]
    ChangeSum* change;
    uint32_t it;
    uint32_t my_graph = kNoGraph;
    bool my_works = false;
    double my_mass = 0.0, my_change = 0.0;

    static __device__ __forceinline__ T zero() { return 0.0; }
    static __device__ __forceinline__ T add(T x, T y) { return x + y; }
    __device__ __forceinline__ bool works(uint32_t g) const {
        return a.stop[g] > it && (it == 0 || !below_tolerance(prev_change[g]));
    }
    __device__ __forceinline__ bool begin(uint32_t g0, uint32_t g1) const {
        for (uint32_t g = g0; g <= g1; ++g)
            if (works(g)) return true;
        return false;
    }
    __device__ __forceinline__ bool want(uint32_t) const { return true; }
    __device__ __forceinline__ T gather(bool p, uint32_t t) const {
        return static_cast<double>(__uint_as_float(ld_if(p, reinterpret_cast<const uint32_t*>(in) + t, 0u)));
    }
    __device__ __forceinline__ void part(uint64_t i, T x) { a.parts[i] = x; }
    __device__ __forceinline__ T parts(uint64_t i) const { return a.parts[i]; }
    // Makes g the lane's graph (its sums so far go out if it was another).
    __device__ __forceinline__ void enter(uint32_t g) {
        if (g == my_graph) return;
        if (my_graph != kNoGraph) spill();
        my_graph = g;
        my_works = works(g);
        my_mass = mass[g];
    }
    __device__ __forceinline__ void spill() {
        add_change(change + my_graph, my_change, a.tolerance, a.scale);
        my_change = 0.0;
    }
    __device__ __forceinline__ float update(uint32_t v, double sum, float tele, float old) {
        const double p = tele;
        const float x = static_cast<float>((1.0 - a.damp) * p + a.damp * (sum + my_mass * p));
        my_change += fabs(static_cast<double>(x) - static_cast<double>(old));
        a.ranks[v] = x;
        return x;
    }
    struct In {
        uint32_t v, g, len;
        float tele, old;
    };
    __device__ __forceinline__ In load(uint32_t r) const {
        return In{__ldg(a.rows.row_vertex + r), __ldg(a.rows.row_graph + r),
                  __ldg(a.rows.row_start + r + 1) - __ldg(a.rows.row_start + r), 0.f, 0.f};
    }
    __device__ __forceinline__ void more(In& x) const {
        x.tele = __ldg(a.tele + x.v);
        x.old = __uint_as_float(ld_if(true, reinterpret_cast<const uint32_t*>(a.ranks) + x.v, 0u));
    }
    __device__ __forceinline__ void finish(uint32_t, T sum, const In& in) {
        enter(in.g);
        if (!my_works) return;
        out[in.v] = update(in.v, sum, in.tele, in.old) / static_cast<float>(in.len);
    }
    __device__ __forceinline__ void finish_lone(uint32_t i) {
        enter(__ldg(a.rows.lone_graph + i));
        if (!my_works) return;
        const uint32_t v = __ldg(a.rows.lone + i);
        update(v, 0.0, a.tele[v], a.ranks[v]);
    }
    __device__ __forceinline__ void flush() {
        const unsigned has = __ballot_sync(kFullMask, my_graph != kNoGraph);
        if (has) {
            // One graph per warp turn nearly always.
            const uint32_t g = __shfl_sync(kFullMask, my_graph, __ffs(has) - 1);
            const bool same = my_graph == g;
            const double part = warp_sum(same ? my_change : 0.0);
            if (lane_id() == static_cast<unsigned>(__ffs(has) - 1)) add_change(change + g, part, a.tolerance, a.scale);
            if (same) my_change = 0.0;
            else if (my_graph != kNoGraph) spill();
        }
        my_graph = kNoGraph;
    }
};

// The dangling mass of the ranks that an iteration makes from the mass before it: a
// vertex without entries gets nothing but its teleport, so its rank follows from
// that mass alone (update() with an empty sum), and is 0 unless it is a seed. A
// group of lanes per graph, in a fixed order.
__device__ __forceinline__ void batch_next_mass(const BatchPpr& a, const double* mass, double* next, uint64_t tid,
                                                uint64_t nthreads) {
    const uint32_t lanes = 1u << a.log_lanes, at = static_cast<uint32_t>(tid) & (lanes - 1);
    for (uint64_t b = (tid & ~31ull) >> a.log_lanes; b < a.G; b += nthreads >> a.log_lanes) {
        const uint64_t g = b + (lane_id() >> a.log_lanes);
        double sum = 0.0;
        if (g < a.G) {
            const double m = mass[g];
            auto rank = [&](double p) {
                return static_cast<double>(static_cast<float>((1.0 - a.damp) * p + a.damp * (0.0 + m * p)));
            };
            for (uint32_t k = at; k < a.K; k += lanes) {
                const float p = __ldg(a.lone_tele + g * a.K + k);
                if (p != 0.f) sum += rank(static_cast<double>(p));
            }
            // The others' rank is 0, or NaN once the mass is no number.
            if (at == 0 && a.lone_count[g] > 0) sum += rank(0.0);
        }
        for (uint32_t d = lanes / 2; d > 0; d /= 2) sum += __shfl_xor_sync(kFullMask, sum, d);
        if (g < a.G && at == 0) next[g] = sum;
    }
}

__global__ void __launch_bounds__(kBatchThreads, kBatchCtasPerSm) batch_ppr_kernel(const BatchPpr a) {
    __shared__ uint32_t s_active;
    __shared__ double s_rows[kBatchThreads / 32][kBatchChunk];
    const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t nthreads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    unsigned barriers = 0;
    auto start = [&](uint32_t g) { return 1.0f / static_cast<float>(a.vbase[g + 1] - a.vbase[g]); };
    for (uint64_t r = tid; r < a.rows.n_rows; r += nthreads) {
        const uint32_t v = a.rows.row_vertex[r];
        const float r0 = start(a.rows.row_graph[r]);
        a.ranks[v] = r0;
        a.contrib_a[v] = r0 / static_cast<float>(a.rows.row_start[r + 1] - a.rows.row_start[r]);
    }
    for (uint64_t i = tid; i < a.rows.n_lone; i += nthreads) {
        // A CSR that is not symmetric may list such a vertex as a target.
        const uint32_t v = a.rows.lone[i];
        a.ranks[v] = start(a.rows.lone_graph[i]);
        a.contrib_a[v] = 0.f;
        a.contrib_b[v] = 0.f;
    }
    for (uint64_t g = tid; g < a.G; g += nthreads) {
        const bool some = a.vbase[g + 1] > a.vbase[g];
        for (uint64_t q = 0; q < 3; ++q) a.change[q * a.G + g] = ChangeSum{0, 0};
        a.mass[g] = some ? static_cast<double>(a.lone_count[g]) * static_cast<double>(start(static_cast<uint32_t>(g))) : 0.0;
        a.stop[g] = some ? 0xFFFFFFFFu : 0u;
    }
    if (!grid_barrier(&a.st->bar, barriers)) return;
    for (uint32_t it = 0; it < a.max_iterations; ++it) {
        const uint64_t cur = static_cast<uint64_t>(it % 3) * a.G, prev = static_cast<uint64_t>((it + 2) % 3) * a.G;
        const uint64_t next = static_cast<uint64_t>((it + 1) % 3) * a.G;
        PprOp op{a, (it & 1) ? a.contrib_b : a.contrib_a, (it & 1) ? a.contrib_a : a.contrib_b,
                 a.change + prev, a.mass + static_cast<uint64_t>(it & 1) * a.G, a.change + cur, it};
        for (uint64_t g = tid; g < a.G; g += nthreads) {
            a.change[next + g] = ChangeSum{0, 0};  // last read an iteration ago
            if (a.stop[g] <= it) continue;
            if (it && below_tolerance(op.prev_change[g])) a.stop[g] = it;
            else atomicAdd(a.st->active + it % 3, 1u);
        }
        batch_next_mass(a, op.mass, a.mass + static_cast<uint64_t>(~it & 1) * a.G, tid, nthreads);
        if (tid == 0) a.st->active[(it + 1) % 3] = 0;
        for (uint64_t b = tid & ~31ull; b < a.rows.n_lone; b += nthreads) {
            if (b + lane_id() < a.rows.n_lone) op.finish_lone(static_cast<uint32_t>(b + lane_id()));
            op.flush();
        }
        batch_pass(a.rows, op, s_rows[threadIdx.x >> 5]);
        if (!grid_barrier(&a.st->bar, gridDim.x, barriers, [&] { s_active = __ldcg(a.st->active + it % 3); })) return;
        if (s_active == 0) break;
        batch_split_pass(a.rows, op);
        if (!grid_barrier(&a.st->bar, barriers)) return;
    }
    // A graph whose last iteration met the tolerance has not been marked yet.
    for (uint64_t g = tid; g < a.G; g += nthreads) {
        uint32_t n = a.stop[g];
        bool conv = n != 0xFFFFFFFFu;
        if (!conv) {
            n = a.max_iterations;
            conv = n > 0 && below_tolerance(a.change[static_cast<uint64_t>((n + 2) % 3) * a.G + g]);
        }
        a.iterations[g] = n;
        a.converged[g] = conv ? 1 : 0;
    }
}

// ---------------------------------------------------------------- host

struct BatchImpl {
    std::shared_ptr<DeviceImpl> dev;
    GraphImpl u;  // the union CSR
    uint32_t G = 0;
    std::vector<uint32_t> vbase, ebase;
    DeviceBuffer<uint32_t> d_vbase;
    // rows of the union for the BFS and PageRank passes (built with the batch)
    BatchRows rows{};
    DeviceBuffer<uint32_t> row_vertex, row_graph, row_start, chunk_row, lone, lone_graph, lone_count;
    DeviceBuffer<uint8_t> delta;
    DeviceBuffer<uint4> split;
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

// vbase uploaded, ebase gathered, the rows of the BFS and PageRank passes.
Error finish_layout(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    const uint32_t G = b.G, V = b.u.num_nodes, E = b.u.num_edges;
    GCU_TRY(b.d_vbase.allocate(dev, G + 1));
    GCU_CUDA(cudaMemcpyAsync(b.d_vbase.ptr, b.vbase.data(), 4 * (G + 1), cudaMemcpyHostToDevice, dev.stream), "copy");
    DeviceBuffer<uint32_t> d_ebase, pos, split_pos;
    GCU_TRY(d_ebase.allocate(dev, G + 1));
    GCU_LAUNCH(dev, "batch_entry_base", batch_entry_base_kernel, small_grid(dev, G + 1, 256), 256, 0, b.u.offsets.ptr,
               b.d_vbase.ptr, G, d_ebase.ptr);
    b.ebase.resize(G + 1);
    GCU_CUDA(cudaMemcpyAsync(b.ebase.data(), d_ebase.ptr, 4 * (G + 1), cudaMemcpyDeviceToHost, dev.stream), "copy");

    GCU_TRY(pos.allocate(dev, static_cast<uint64_t>(V) + 1));
    if (V)
        GCU_LAUNCH(dev, "batch_row_flags", batch_row_flags_kernel, small_grid(dev, V, 256), 256, 0, b.u.offsets.ptr, V,
                   pos.ptr);
    GCU_TRY(exclusive_scan_u32(dev, pos.ptr, pos.ptr, V));
    uint32_t n_rows = 0;
    GCU_CUDA(cudaMemcpyAsync(&n_rows, pos.ptr + V, sizeof(uint32_t), cudaMemcpyDeviceToHost, dev.stream), "copy");
    GCU_TRY(dev.sync());
    const uint32_t n_chunks = static_cast<uint32_t>(ceil_div_u64(E, kBatchChunk));
    GCU_TRY(b.row_vertex.allocate(dev, n_rows));
    GCU_TRY(b.row_graph.allocate(dev, n_rows));
    GCU_TRY(b.row_start.allocate(dev, static_cast<uint64_t>(n_rows) + 1));
    GCU_TRY(b.lone.allocate(dev, V - n_rows));
    GCU_TRY(b.lone_graph.allocate(dev, V - n_rows));
    GCU_TRY(b.lone_count.allocate(dev, std::max<uint32_t>(G, 1)));
    GCU_CUDA(cudaMemsetAsync(b.lone_count.ptr, 0, 4ull * std::max<uint32_t>(G, 1), dev.stream), "memset");
    GCU_LAUNCH(dev, "batch_rows", batch_rows_kernel, small_grid(dev, static_cast<uint64_t>(V) + 1, 256), 256, 0,
               b.u.offsets.ptr, pos.ptr, b.d_vbase.ptr, G, V, E, b.row_vertex.ptr, b.row_graph.ptr, b.row_start.ptr,
               b.lone.ptr, b.lone_graph.ptr, b.lone_count.ptr);
    GCU_TRY(b.chunk_row.allocate(dev, n_chunks));
    GCU_TRY(b.delta.allocate(dev, static_cast<uint64_t>(n_chunks) * kBatchChunk));
    uint32_t n_split = 0;
    if (n_rows) {
        GCU_TRY(split_pos.allocate(dev, static_cast<uint64_t>(n_rows) + 1));
        GCU_LAUNCH(dev, "batch_chunk_rows", batch_chunk_rows_kernel, small_grid(dev, n_rows, 256), 256, 0,
                   b.row_start.ptr, n_rows, b.chunk_row.ptr, split_pos.ptr);
        GCU_TRY(exclusive_scan_u32(dev, split_pos.ptr, split_pos.ptr, n_rows));
        GCU_CUDA(cudaMemcpyAsync(&n_split, split_pos.ptr + n_rows, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                 dev.stream),
                 "copy");
        GCU_CUDA(cudaMemsetAsync(b.delta.ptr, 0, static_cast<size_t>(n_chunks) * kBatchChunk, dev.stream), "memset");
        GCU_LAUNCH(dev, "batch_delta", batch_delta_kernel, small_grid(dev, E, 1024), 256, 0, b.row_start.ptr, n_rows,
                   E, b.chunk_row.ptr, b.delta.ptr);
        GCU_TRY(dev.sync());
    }
    GCU_TRY(b.split.allocate(dev, n_split));
    if (n_split)
        GCU_LAUNCH(dev, "batch_split_rows", batch_split_rows_kernel, small_grid(dev, n_rows, 256), 256, 0,
                   b.row_start.ptr, n_rows, split_pos.ptr, b.split.ptr);
    b.rows = BatchRows{b.u.targets.ptr, b.row_vertex.ptr, b.row_graph.ptr, b.row_start.ptr, b.chunk_row.ptr,
                       b.delta.ptr, b.split.ptr, b.lone.ptr, b.lone_graph.ptr, E, n_rows, n_chunks, n_split,
                       V - n_rows};
    // Zero until a pass kernel runs: results may be read before.
    for (auto* st : {&b.bfs_state, &b.ppr_state}) {
        GCU_TRY(st->allocate(dev, 1));
        GCU_CUDA(cudaMemsetAsync(st->ptr, 0, sizeof(BatchRunState), dev.stream), "memset");
    }
    return dev.sync();
}

// Blocks of a pass kernel: all that are resident at once, fewer for a batch
// too small to give every warp a turn.
template <class Kernel>
Error pass_grid(BatchImpl& b, Kernel kernel, unsigned* grid) {
    if (*grid) return ok();
    int per_sm = 0;
    GCU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBatchThreads, 0), "occupancy");
    const uint64_t most = static_cast<uint64_t>(b.dev->sm_count) * std::max(1, std::min(per_sm, kBatchCtasPerSm));
    const uint64_t want = std::max<uint64_t>({1, ceil_div_u64(b.rows.n_chunks, kBatchThreads / 32),
                                              ceil_div_u64(b.u.num_nodes, 4 * kBatchThreads)});
    *grid = static_cast<unsigned>(std::min(want, most));
    return ok();
}

Error launch_bfs(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    GCU_TRY(pass_grid(b, batch_bfs_kernel, &b.bfs_grid));
    if (b.keep_dist)
        GCU_CUDA(cudaMemsetAsync(b.dist.ptr, 0xFF, sizeof(int32_t) * b.S * static_cast<size_t>(b.u.num_nodes),
                                 dev.stream),
                 "memset");
    GCU_CUDA(cudaMemsetAsync(b.bfs_state.ptr, 0, sizeof(BatchRunState), dev.stream), "memset");
    BatchBfs a{};
    a.rows = b.rows;
    a.offsets = b.u.offsets.ptr;
    a.vbase = b.d_vbase.ptr;
    a.sources = b.sources.ptr;
    a.G = b.G;
    a.V = b.u.num_nodes;
    a.S = b.S;
    a.full = b.S >= 32 ? 0xFFFFFFFFu : (1u << b.S) - 1u;
    a.mask_a = b.mask_a.ptr;
    a.mask_b = b.mask_b.ptr;
    a.parts = b.bfs_parts.ptr;
    a.dist = b.keep_dist ? b.dist.ptr : nullptr;
    a.fresh = b.fresh.ptr;
    a.stop = b.bfs_stop.ptr;
    a.reachable = b.reachable.ptr;
    a.max_depth = b.max_depth.ptr;
    a.st = b.bfs_state.ptr;
    GCU_LAUNCH_COOP(dev, "batch_bfs", batch_bfs_kernel, b.bfs_grid, kBatchThreads, 0, a);
    return ok();
}

Error launch_ppr(BatchImpl& b) {
    DeviceImpl& dev = *b.dev;
    GCU_TRY(pass_grid(b, batch_ppr_kernel, &b.ppr_grid));
    GCU_CUDA(cudaMemsetAsync(b.ppr_state.ptr, 0, sizeof(BatchRunState), dev.stream), "memset");
    BatchPpr a{};
    a.rows = b.rows;
    a.vbase = b.d_vbase.ptr;
    a.lone_count = b.lone_count.ptr;
    a.tele = b.tele.ptr;
    a.lone_tele = b.lone_tele.ptr;
    a.G = b.G;
    a.V = b.u.num_nodes;
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
    return ok();
}

// Reads a pass kernel's error flag (the stream has been synchronized).
Error check_run(BatchImpl& b, const DeviceBuffer<BatchRunState>& st, const char* what) {
    BatchRunState h{};
    GCU_CUDA(cudaMemcpyAsync(&h, st.ptr, sizeof(h), cudaMemcpyDeviceToHost, b.dev->stream), "copy");
    GCU_TRY(b.dev->sync());
    if (h.bar.failed) return kernel_error(std::string(what) + ": a block did not reach the grid barrier");
    return ok();
}

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
    const uint64_t V = b.u.num_nodes;
    b.S = S;
    b.keep_dist = keep_distances;
    GCU_TRY(b.sources.allocate(dev, static_cast<uint64_t>(b.G) * S));
    GCU_CUDA(cudaMemcpyAsync(b.sources.ptr, sources, 4ull * b.G * S, cudaMemcpyHostToDevice, dev.stream), "copy");
    GCU_TRY(b.bfs_parts.allocate(dev, 2ull * b.rows.n_chunks));
    GCU_TRY(b.fresh.allocate(dev, 3ull * b.G));
    GCU_TRY(b.bfs_stop.allocate(dev, b.G));
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
    const uint64_t V = b.u.num_nodes;
    b.K = K;
    b.damping = damping;
    b.max_iterations = max_iterations;
    b.tolerance = tolerance;
    GCU_TRY(b.seeds.allocate(dev, static_cast<uint64_t>(b.G) * K));
    GCU_CUDA(cudaMemcpyAsync(b.seeds.ptr, seeds, 4ull * b.G * K, cudaMemcpyHostToDevice, dev.stream), "copy");
    GCU_TRY(b.tele.allocate(dev, V));
    GCU_TRY(b.ppr_parts.allocate(dev, 2ull * b.rows.n_chunks));
    GCU_TRY(b.change.allocate(dev, 3ull * b.G));
    GCU_TRY(b.mass.allocate(dev, 2ull * b.G));
    GCU_TRY(b.lone_tele.allocate(dev, static_cast<uint64_t>(b.G) * K));
    GCU_TRY(b.ppr_stop.allocate(dev, b.G));
    GCU_TRY(b.contrib_a.allocate(dev, V));
    GCU_TRY(b.contrib_b.allocate(dev, V));
    GCU_TRY(b.ranks.allocate(dev, V));
    GCU_TRY(b.iterations.allocate(dev, std::max<uint32_t>(b.G, 1)));
    GCU_TRY(b.converged.allocate(dev, std::max<uint32_t>(b.G, 1)));
    GCU_CUDA(cudaMemsetAsync(b.tele.ptr, 0, 4 * std::max<uint64_t>(V, 1), dev.stream), "memset");
    GCU_LAUNCH(dev, "batch_tele", batch_tele_kernel, small_grid(dev, static_cast<uint64_t>(b.G) * K, 256), 256, 0,
               b.seeds.ptr, b.d_vbase.ptr, b.G, K, b.tele.ptr);
    // Each graph's seeds once, in order, then their teleports where they have no entries.
    std::vector<uint32_t> once(seeds, seeds + static_cast<uint64_t>(b.G) * K);
    for (uint32_t g = 0; g < b.G; ++g) {
        const auto first = once.begin() + static_cast<int64_t>(g) * K, last = first + K;
        std::sort(first, last);
        std::fill(std::unique(first, last), last, kNoSeed);
    }
    GCU_CUDA(cudaMemcpyAsync(b.seeds.ptr, once.data(), 4ull * b.G * K, cudaMemcpyHostToDevice, dev.stream), "copy");
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
    GCU_TRY(check_run(b, b.bfs_state, "batch BFS"));
    if (distances && b.keep_dist) GCU_TRY(copy_to_host(dev, distances, b.dist.ptr, 4ull * b.S * b.u.num_nodes));
    if (reachable) GCU_CUDA(cudaMemcpyAsync(reachable, b.reachable.ptr, 4 * gs, cudaMemcpyDeviceToHost, dev.stream), "copy");
    if (max_depth) GCU_CUDA(cudaMemcpyAsync(max_depth, b.max_depth.ptr, 4 * gs, cudaMemcpyDeviceToHost, dev.stream), "copy");
    return dev.sync();
}

Error batch_read_ppr(BatchImpl& b, float* ranks, uint32_t* iterations, uint8_t* converged) {
    DeviceImpl& dev = *b.dev;
    GCU_TRY(check_run(b, b.ppr_state, "batch PageRank"));
    if (ranks) GCU_TRY(copy_to_host(dev, ranks, b.ranks.ptr, 4ull * b.u.num_nodes));
    if (iterations)
        GCU_CUDA(cudaMemcpyAsync(iterations, b.iterations.ptr, 4ull * b.G, cudaMemcpyDeviceToHost, dev.stream), "copy");
    if (converged)
        GCU_CUDA(cudaMemcpyAsync(converged, b.converged.ptr, b.G, cudaMemcpyDeviceToHost, dev.stream), "copy");
    return dev.sync();
}

// Captures triangle counts, BFS and PageRank of the whole batch into one CUDA
// graph (plans and autotunes first: nothing in the capture allocates or syncs).
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

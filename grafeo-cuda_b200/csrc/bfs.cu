// Breadth-first search: direction-optimising, level synchronous.
//
// Reference: crates/grafeo-cuda-algos/src/bfs.rs:42-131 and kernels/bfs.cu:54-83
// (one thread per frontier vertex walking its whole list, an atomicCAS per
// edge on `distances`, one global atomic per discovered vertex, and a host
// sync plus a 4-byte copy per level). Here:
//
//  * Top-down step (small frontiers): the frontier's edges are split evenly
//    over blocks (an exclusive scan of frontier degrees, then a load-balanced
//    search per block over the scan staged in shared memory), so a hub's list
//    is read by many blocks with coalesced loads instead of one thread.
//    Discovery is an atomicOr on a visited bitmap (V/8 bytes, L2 resident)
//    after a plain test; the next queue is appended with one atomic per warp.
//  * Bottom-up step (large frontiers, symmetric graphs only): every unvisited
//    vertex scans its list for a parent in the frontier bitmap and stops at the
//    first hit (Beamer, Asanovic and Patterson, SC'12). No atomics: each warp
//    owns one bitmap word of 32 vertices; a lane checks the first entries of
//    its vertex's list alone and longer lists are walked by the whole warp,
//    32 coalesced entries per step.
//  * Three step variants: push with one warp per frontier vertex (one
//    launch), load-balanced push (above), pull (above).
//  * One launch per search (bfs_search_kernel) under the fixed schedule; a graph
//    of conditional nodes over the step kernels under a learned one.
//  * Schedule: Beamer's alpha/beta rule (alpha = 14, beta = 24) over the
//    balanced push and the pull, fed by the frontier and unexplored edge
//    counts the steps emit; or, when a learned schedule is installed on the
//    device, a one-warp kernel after every step that turns the step's
//    counters into features and picks the variant with the smallest predicted
//    time (sched.cuh), with the alpha/beta rule as its fallback. The schedule
//    only changes which kernels run; BFS levels are unique, so the distances
//    cannot change.
//  * Trace mode (bfs_trace) times every valid variant at every level from the
//    same frontier: the training data of the learned schedule.
//  * Vertices without out-edges are counted and labelled but never queued.
#include <algorithm>

#include "device_common.cuh"
#include "gcu_internal.h"
#include "sched.cuh"

namespace gcu {

constexpr int kTdThreads = 256;
constexpr int kTdItems = 4;
constexpr int kTdTile = kTdThreads * kTdItems;  // frontier edges per block
constexpr int kBuThreads = 256;

struct BfsCounters {
    uint32_t discovered;  // vertices labelled this level
    uint32_t queued;      // of those, vertices with out-edges (appended to the queue)
    unsigned long long edges;  // sum of out-degrees of the vertices labelled this level
    int32_t choice;       // learned schedule's variant for the next step (-1: use the fixed rule)
    uint32_t pad;
};

// Step variants (the learned schedule's three outputs for a BFS level).
enum BfsVariant : int {
    kPushWarp = 0,      // top-down, one warp per frontier vertex, one launch
    kPushBalanced = 1,  // top-down, frontier edges split evenly over blocks (degrees + scan + expand)
    kPull = 2,          // bottom-up over the frontier bitmap (symmetric graphs only)
};

// Where a device-driven run stands between two steps (the device twin of the
// host loop's BfsState, kept in device memory and read by every step kernel).
struct BfsDevState {
    unsigned long long frontier_m;  // out-edges of the frontier
    unsigned long long unexplored;  // out-edges of vertices not labelled yet
    uint32_t frontier_n;            // vertices labelled by the last step
    uint32_t frontier_q;            // of those, queued (out-degree > 0)
    uint32_t reached;
    int32_t level;                  // level of the frontier
    uint32_t cur;                   // queue[cur] / bitmap[cur] hold the frontier
    uint32_t bitmap_valid;          // the last step was a pull: bitmap[cur] holds the frontier
    int32_t variant;                // the step the SWITCH node runs next (kSchedOut: none)
    uint32_t first;                 // the counters are the source's, not a step's
    uint32_t failed;                // the loop stopped on a state no search can reach
};

struct BfsSearchState;

struct BfsWork {
    DeviceBuffer<int32_t> dist;
    DeviceBuffer<uint32_t> visited;
    int symmetric = -1;                    // -1 unknown, 0 no, 1 yes
    DeviceBuffer<uint32_t> active;         // vertices with edges, ascending (symmetric graphs)
    uint32_t n_active = 0;
    bool pull_list = false;                // the pull walks `active` instead of every bitmap word
    // one-launch search (ensure_search)
    bool search_ready = false;
    DeviceBuffer<uint32_t> search_bitmaps;  // three
    DeviceBuffer<uint2> items[2];
    DeviceBuffer<uint4> search_segments;
    uint32_t search_epoch = 0;
    DeviceBuffer<BfsSearchState> search;
    unsigned search_grid = 0;
    struct {
        uint32_t reached;
        int32_t level;
        uint32_t failed;
    } host_search{};
    // level by level, driven by the device or the host, and the trace (ensure_levels)
    bool levels_ready = false;
    DeviceBuffer<uint32_t> bitmap[2];
    DeviceBuffer<uint32_t> queue[2];
    DeviceBuffer<uint32_t> degree_scan;  // V + 1
    DeviceBuffer<BfsCounters> counters;
    BfsCounters host_counters{};  // host copy, read after a synchronisation (plain memory)
    // device-driven level loop (built on first use, per schedule network)
    DeviceBuffer<BfsDevState> loop_state;
    DeviceBuffer<uint32_t> loop_scan_sums;
    BfsDevState host_loop_state{};  // host copy of the loop's final state (plain memory)
    cudaGraph_t loop_graph = nullptr;
    cudaGraphExec_t loop_exec = nullptr;
    const void* loop_net = nullptr;  // the schedule network the graph reads (NULL: fixed rule)
    bool loop_unavailable = false;   // the driver refused the graph: the host drives the levels
};

void destroy_bfs_work(BfsWork* w) {
    if (!w) return;
    if (w->loop_exec) cudaGraphExecDestroy(w->loop_exec);
    if (w->loop_graph) cudaGraphDestroy(w->loop_graph);
    delete w;
}

// ---------------------------------------------------------------- kernels

__device__ __forceinline__ void append_warp(bool take, uint32_t v, uint32_t* __restrict__ queue,
                                            uint32_t* __restrict__ count) {
    const unsigned mask = __ballot_sync(kFullMask, take);
    if (mask == 0) return;
    const unsigned lane = lane_id();
    uint32_t base = 0;
    if (lane == static_cast<unsigned>(__ffs(mask) - 1)) base = atomicAdd(count, static_cast<uint32_t>(__popc(mask)));
    base = __shfl_sync(kFullMask, base, __ffs(mask) - 1);
    if (take) queue[base + __popc(mask & ((1u << lane) - 1))] = v;
}

// Per-lane totals of what a lane labelled; a warp adds them to the level's
// counters once, when it is done (flush_tally), instead of one atomic pair on
// the same two words per warp step.
struct Tally {
    uint32_t found = 0;
    unsigned long long edges = 0;
};

// Labels v (found by a parent at this level) and records it; called by all
// lanes of a warp, `found` says whether this lane discovered a vertex.
__device__ __forceinline__ void record_discovery(bool found, uint32_t v, const uint32_t* __restrict__ offsets,
                                                 int32_t* __restrict__ dist, int32_t level,
                                                 uint32_t* __restrict__ next_queue, BfsCounters* __restrict__ ctr,
                                                 Tally& tally) {
    uint32_t deg = 0;
    if (found) {
        dist[v] = level;
        deg = offsets[v + 1] - offsets[v];
        tally.found += 1;
        tally.edges += deg;
    }
    if (__ballot_sync(kFullMask, found) == 0) return;
    append_warp(found && deg > 0, v, next_queue, &ctr->queued);
}

// All 32 lanes call it once, at the end of the kernel.
__device__ __forceinline__ void flush_tally(const Tally& tally, BfsCounters* __restrict__ ctr) {
    const uint32_t found = warp_sum(tally.found);
    const unsigned long long edges = warp_sum(tally.edges);
    if (lane_id() == 0) {
        if (found) atomicAdd(&ctr->discovered, found);
        if (edges) atomicAdd(&ctr->edges, edges);
    }
}

__global__ void bfs_init_kernel(const uint32_t* __restrict__ offsets, uint32_t source, int32_t* __restrict__ dist,
                                uint32_t* __restrict__ visited, uint32_t* __restrict__ queue,
                                BfsCounters* __restrict__ ctr) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    dist[source] = 0;
    visited[source >> 5] |= 1u << (source & 31);
    uint32_t deg = offsets[source + 1] - offsets[source];
    queue[0] = source;
    ctr->discovered = 1;
    ctr->queued = deg > 0 ? 1 : 0;
    ctr->edges = deg;
}

__global__ void bfs_queue_degrees_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ queue,
                                         uint32_t n, uint32_t* __restrict__ deg) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        uint32_t u = queue[i];
        deg[i] = offsets[u + 1] - offsets[u];
    }
}

// Top-down: the block expands frontier edges [e0, e0 + kTdTile) of `total`
// (every thread of the block calls it with the same tile).
__device__ __forceinline__ void topdown_tile(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets,
                                             const uint32_t* __restrict__ queue, uint32_t qsize,
                                             const uint32_t* __restrict__ qscan, uint32_t total, uint64_t e0,
                                             int32_t* __restrict__ dist, uint32_t* __restrict__ visited,
                                             uint32_t* __restrict__ next_queue, BfsCounters* __restrict__ ctr,
                                             int32_t next_level, Tally& tally) {
    __shared__ uint32_t s_scan[kTdTile + 1];
    __shared__ uint32_t s_start[kTdTile + 1];
    __shared__ uint32_t s_range[2];
    const uint32_t e1 = static_cast<uint32_t>(min_u64(e0 + kTdTile, total));
    if (threadIdx.x < 2) {
        // Largest frontier index i with qscan[i] <= e (each queued vertex owns >= 1 edge).
        uint32_t e = threadIdx.x == 0 ? static_cast<uint32_t>(e0) : e1 - 1;
        uint32_t lo = 0, hi = qsize;
        while (hi - lo > 1) {
            uint32_t mid = lo + ((hi - lo) >> 1);
            if (qscan[mid] <= e)
                lo = mid;
            else
                hi = mid;
        }
        s_range[threadIdx.x] = lo;
    }
    __syncthreads();
    const uint32_t i0 = s_range[0];
    const uint32_t window = s_range[1] - i0 + 1;  // <= kTdTile
    for (uint32_t k = threadIdx.x; k < window; k += kTdThreads) {
        s_scan[k] = qscan[i0 + k];
        s_start[k] = offsets[queue[i0 + k]];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kTdItems; ++q) {
        const uint32_t o = q * kTdThreads + threadIdx.x, e = static_cast<uint32_t>(e0) + o;
        bool found = false;
        uint32_t v = 0;
        if (o < e1 - static_cast<uint32_t>(e0)) {
            uint32_t lo = 0, hi = window;
            while (hi - lo > 1) {
                uint32_t mid = (lo + hi) >> 1;
                if (s_scan[mid] <= e)
                    lo = mid;
                else
                    hi = mid;
            }
            v = ld_stream(targets + s_start[lo] + (e - s_scan[lo]));
            const uint32_t bit = 1u << (v & 31);
            if (!(__ldcg(visited + (v >> 5)) & bit)) found = !(atomicOr(visited + (v >> 5), bit) & bit);
        }
        record_discovery(found, v, offsets, dist, next_level, next_queue, ctr, tally);
    }
}

// Top-down: block b expands frontier edges [b*kTdTile, (b+1)*kTdTile).
__global__ void __launch_bounds__(kTdThreads) bfs_topdown_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, const uint32_t* __restrict__ queue,
    uint32_t qsize, const uint32_t* __restrict__ qscan, int32_t* __restrict__ dist, uint32_t* __restrict__ visited,
    uint32_t* __restrict__ next_queue, BfsCounters* __restrict__ ctr, int32_t next_level) {
    const uint32_t total = qscan[qsize];
    const uint64_t e0 = static_cast<uint64_t>(blockIdx.x) * kTdTile;
    if (e0 >= total) return;
    Tally tally;
    topdown_tile(offsets, targets, queue, qsize, qscan, total, e0, dist, visited, next_queue, ctr, next_level, tally);
    flush_tally(tally, ctr);
}

__global__ void bfs_queue_to_bitmap_kernel(const uint32_t* __restrict__ queue, uint32_t n,
                                           uint32_t* __restrict__ bitmap) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        uint32_t u = queue[i];
        atomicOr(bitmap + (u >> 5), 1u << (u & 31));
    }
}

constexpr uint32_t kBuSolo = 8;  // entries a lane checks alone before its warp takes over the list
// The pull step walks the list of vertices with edges when at least
// 1 / kBuListFraction of the vertices are isolated (R-MAT 22: 43 %; list
// 7.5 % faster than the word form there, 10 % at R-MAT 24), and every word of
// the visited bitmap otherwise (Erdos-Renyi 2^22, almost no isolated vertex:
// the word form is 9 % faster, without the list's atomics and indirection).
constexpr uint32_t kBuListFraction = 8;

__device__ __forceinline__ bool in_frontier(const uint32_t* __restrict__ frontier, uint32_t u) {
    return (__ldg(frontier + (u >> 5)) >> (u & 31)) & 1u;
}

// Bottom-up: warp w handles the 32 vertices of bitmap word w. Each unvisited
// vertex first checks its first kBuSolo entries alone (4 loads in flight);
// most vertices that have a parent in a large frontier find it there. The
// lists that are left are then walked by the whole warp, one list at a time,
// 32 consecutive entries per step (coalesced) with a ballot to stop at the
// first parent, so a long list neither serialises one lane nor stalls the
// other 31.
// Whether this lane's vertex (list [s, e); e == s: nothing to probe) has a
// neighbour in the frontier. Called by all 32 lanes: the lists left after
// the solo probes are walked by the whole warp.
__device__ __forceinline__ bool probe_parent(uint32_t s, uint32_t e, const uint32_t* __restrict__ frontier,
                                             const uint32_t* __restrict__ targets) {
    const unsigned lane = lane_id();
    bool found = false;
    const uint32_t solo = min(e - s, kBuSolo);
    for (uint32_t k = 0; k < solo && !found; k += 4) {
        uint32_t t[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) t[q] = k + q < solo ? targets[s + k + q] : 0xFFFFFFFFu;
#pragma unroll
        for (int q = 0; q < 4; ++q) found = found || (t[q] != 0xFFFFFFFFu && in_frontier(frontier, t[q]));
    }
    unsigned pending = __ballot_sync(kFullMask, !found && e - s > kBuSolo);
    while (pending) {
        const int p = __ffs(pending) - 1;
        pending &= pending - 1;
        const uint64_t ps = static_cast<uint64_t>(__shfl_sync(kFullMask, s, p)) + kBuSolo;
        const uint64_t pe = __shfl_sync(kFullMask, e, p);
        bool hit = false;
        for (uint64_t base = ps; base < pe; base += 32) {
            const uint64_t j = base + lane;
            const bool h = j < pe && in_frontier(frontier, targets[j]);
            if (__ballot_sync(kFullMask, h)) {
                hit = true;
                break;
            }
        }
        if (static_cast<int>(lane) == p) found = hit;
    }
    return found;
}

// Word form: warp w handles the 32 vertices of bitmap word w (it owns that
// word of `visited` and writes the word of `next_frontier`, found or not).
__device__ __forceinline__ void bottomup_body(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, uint32_t V,
    const uint32_t* __restrict__ frontier, uint32_t* __restrict__ next_frontier, uint32_t* __restrict__ visited,
    int32_t* __restrict__ dist, uint32_t* __restrict__ next_queue, BfsCounters* __restrict__ ctr,
    int32_t next_level) {
    const unsigned lane = lane_id();
    const uint64_t words = ceil_div_u64(V, 32);
    const uint64_t warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    Tally tally;
    for (uint64_t w = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < words; w += warps) {
        // The word's visited bits and its lanes' list bounds, loaded side by
        // side (the bounds of visited vertices are read too, then ignored).
        const uint32_t vis = visited[w];
        const uint32_t v = static_cast<uint32_t>(w * 32 + lane);
        uint32_t s = 0, e = 0;
        if (v < V) {
            s = offsets[v];
            e = offsets[v + 1];
        }
        const bool open = v < V && !((vis >> lane) & 1u);
        if (!open) e = s;
        const bool found = probe_parent(s, e, frontier, targets);
        const unsigned mask = __ballot_sync(kFullMask, found);
        if (lane == 0) {
            next_frontier[w] = mask;
            if (mask) visited[w] = vis | mask;
        }
        record_discovery(found, v, offsets, dist, next_level, next_queue, ctr, tally);
    }
    flush_tally(tally, ctr);
}

// List form: the warps stride over the graph's vertices with edges (`active`,
// ascending), 32 at a time, so no lane sits on an isolated vertex (43 % of
// R-MAT 22's). A word of the bitmaps can span two warps' batches, so found
// vertices set their bits with atomicOr; the caller clears next_frontier.
__device__ __forceinline__ void bottomup_list_body(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets,
    const uint32_t* __restrict__ active, uint32_t n_active, const uint32_t* __restrict__ frontier,
    uint32_t* __restrict__ next_frontier, uint32_t* visited, int32_t* __restrict__ dist,
    uint32_t* __restrict__ next_queue, BfsCounters* __restrict__ ctr, int32_t next_level) {
    const unsigned lane = lane_id();
    const uint64_t warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    Tally tally;
    for (uint64_t base = ((static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * 32; base < n_active;
         base += warps * 32) {
        const uint64_t i = base + lane;
        uint32_t v = 0, s = 0, e = 0;
        bool open = false;
        if (i < n_active) {
            v = active[i];
            // Only this lane sets its vertex's bit, so a word another warp is
            // updating still shows this bit as it is.
            const uint32_t vis = visited[v >> 5];
            s = offsets[v];
            e = offsets[v + 1];
            open = !((vis >> (v & 31)) & 1u);
        }
        if (!open) e = s;
        const bool found = probe_parent(s, e, frontier, targets);
        if (found) {
            const uint32_t bit = 1u << (v & 31);
            atomicOr(next_frontier + (v >> 5), bit);
            atomicOr(visited + (v >> 5), bit);
        }
        record_discovery(found, v, offsets, dist, next_level, next_queue, ctr, tally);
    }
    flush_tally(tally, ctr);
}

// One instantiation per pull form (kList: walk `active`; else every bitmap
// word), so that each keeps its own body's register count: the word form
// needs 32 registers, a kernel holding both bodies 38, which costs a quarter
// of the resident warps of whichever form runs.
template <bool kList>
__global__ void __launch_bounds__(kBuThreads) bfs_bottomup_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, uint32_t V,
    const uint32_t* __restrict__ active, uint32_t n_active, const uint32_t* __restrict__ frontier,
    uint32_t* __restrict__ next_frontier, uint32_t* __restrict__ visited, int32_t* __restrict__ dist,
    uint32_t* __restrict__ next_queue, BfsCounters* __restrict__ ctr, int32_t next_level) {
    if (kList)
        bottomup_list_body(offsets, targets, active, n_active, frontier, next_frontier, visited, dist, next_queue, ctr,
                           next_level);
    else
        bottomup_body(offsets, targets, V, frontier, next_frontier, visited, dist, next_queue, ctr, next_level);
}

// Top-down, one warp per frontier vertex (no degree scan: one launch, for
// frontiers whose edges are few or evenly spread).
__device__ __forceinline__ void topdown_warp_body(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, const uint32_t* __restrict__ queue,
    uint32_t qsize, int32_t* __restrict__ dist, uint32_t* __restrict__ visited, uint32_t* __restrict__ next_queue,
    BfsCounters* __restrict__ ctr, int32_t next_level) {
    const unsigned lane = lane_id();
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    Tally tally;
    for (uint64_t i = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; i < qsize; i += nwarps) {
        const uint32_t u = queue[i];
        const uint64_t s = offsets[u], e = offsets[u + 1];
        for (uint64_t b = s; b < e; b += 32) {
            const uint64_t j = b + lane;
            bool found = false;
            uint32_t v = 0;
            if (j < e) {
                v = ld_stream(targets + j);
                const uint32_t bit = 1u << (v & 31);
                if (!(__ldcg(visited + (v >> 5)) & bit)) found = !(atomicOr(visited + (v >> 5), bit) & bit);
            }
            record_discovery(found, v, offsets, dist, next_level, next_queue, ctr, tally);
        }
    }
    flush_tally(tally, ctr);
}

__global__ void __launch_bounds__(kTdThreads) bfs_topdown_warp_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, const uint32_t* __restrict__ queue,
    uint32_t qsize, int32_t* __restrict__ dist, uint32_t* __restrict__ visited, uint32_t* __restrict__ next_queue,
    BfsCounters* __restrict__ ctr, int32_t next_level) {
    topdown_warp_body(offsets, targets, queue, qsize, dist, visited, next_queue, ctr, next_level);
}

// Beamer's direction-optimising thresholds (Beamer, Asanovic and Patterson,
// SC'12): pull when the frontier's edges exceed the unexplored edges / alpha,
// back to push when the frontier falls below V / beta.
constexpr int kAlpha = 14;
constexpr int kBeta = 24;

// Beamer's direction rule over the balanced push and the pull, from the
// state after a step: the fixed schedule, the fallback of the learned one,
// and the variant the learned pick has to beat by a margin.
__host__ __device__ __forceinline__ int bfs_fixed_variant(bool symmetric, bool bottom_up, uint64_t frontier_n,
                                                          uint64_t frontier_m, uint64_t unexplored, uint32_t V) {
    const double alpha = kAlpha, beta = kBeta;
    if (!symmetric) return kPushBalanced;
    if (!bottom_up && static_cast<double>(frontier_m) > static_cast<double>(unexplored) / alpha) return kPull;
    if (bottom_up && static_cast<double>(frontier_n) < static_cast<double>(V) / beta) return kPushBalanced;
    return bottom_up ? kPull : kPushBalanced;
}

// One warp: the features of the decision before expanding the frontier the
// last step produced (its counters, plus the host's totals before that step),
// written to features_out when given; with a network, the chosen variant goes
// to ctr->choice for the host to read with the counters.
__global__ void bfs_decide_kernel(const __nv_bfloat16* __restrict__ w, BfsCounters* __restrict__ ctr,
                                  DegreeStats stats, unsigned long long prior_unexplored, uint32_t prior_reached,
                                  int32_t frontier_level, int frontier_bitmap, unsigned valid_mask, uint32_t num_nodes,
                                  float* __restrict__ features_out) {
    const BfsCounters c = *ctr;
    float f[kSchedIn];
    bfs_features(f, static_cast<float>(c.discovered), static_cast<float>(c.edges),
                 static_cast<float>(prior_unexplored - c.edges), frontier_level, stats, frontier_bitmap != 0,
                 static_cast<float>(prior_reached + c.discovered));
    if (features_out && lane_id() == 0)
        for (int k = 0; k < kSchedIn; ++k) features_out[k] = f[k];
    if (w) {
        float out[kSchedOut];
        sched_forward_warp(w, f, out);
        const int fixed = bfs_fixed_variant((valid_mask >> kPull) & 1u, frontier_bitmap != 0, c.discovered, c.edges,
                                            prior_unexplored - c.edges, num_nodes);
        if (lane_id() == 0) ctr->choice = sched_pick_over(out, valid_mask, fixed);
    }
}

// ---------------------------------------------------------------- one launch per search
//
// The fixed schedule's search runs as one cooperative kernel: every block
// holds the level loop's state in registers and the blocks meet at a grid
// barrier (about 1.5 us) between levels, instead of a graph of conditional
// nodes with four to six launches per level (about 25-30 us per level,
// whatever the frontier's size).
//  * Push levels work on items: ranges of at most kItemEdges list entries of
//    the frontier's vertices, appended when a vertex is discovered. A hub is
//    many items, so the edges are spread evenly with no degree scan; a warp
//    takes up to 32 items at a time and walks their edges in order, found by
//    a search over a warp scan of the item lengths.
//  * While the frontier has at most kLocalEdges edges, block 0 runs the levels
//    alone with its queue in shared memory and block barriers; up to
//    kGroupEdges, the first kGroupBlocks blocks run them with a barrier of
//    their own. A level there is a chain of dependent accesses (317 cycles for
//    an L2 read, 511 for an atomic, measured), and one SM completes one
//    scattered L2 access per cycle, so a frontier of thousands of edges wants
//    a few SMs and a cheap barrier, not one SM and not all.
//  * Pull levels keep no queue: a push that follows builds its items from the
//    frontier bitmap, a pull that follows a push builds the bitmap from the
//    distances (one coalesced pass, far below the level's own work).
// Measured on one B200, a whole search through the Python module (the graph of
// conditional nodes before, this kernel after): R-MAT 14 with distances 195 ->
// 83 us; 1024 x 1024 grid with dropped edges, 1,640 levels, 56.7 -> 5.4 ms (a
// level 31 -> 2.8 us: 1.7 of work, 0.9 of barrier); 16 searches of R-MAT 22
// 9.33 -> 4.18 ms (one: init 9, pushes 14, bitmap 6, pulls 50 + 28 + 15, tail
// 15 us). The same levels with block 0 alone: 5.4 us at 4,000 frontier edges,
// 2.2 at 100, hence kLocalEdges. What bounds it: the levels' latency chains on
// small frontiers, the L1's tag lookups of the pull's scattered probes on wide
// ones (about 130 lookups per 32 vertices; reading a list's sector in one
// 32-byte load and joining the bitmap atomics per word took a third away).
// Level counters rotate over three slots: phase p adds into slot p % 3, reads
// it after its barrier, and clears slot (p + 1) % 3, whose readers are done.
constexpr int kSearchThreads = 1024;
constexpr int kSearchCtasPerSm = 1;
constexpr uint32_t kItemEdges = 1024;
constexpr uint32_t kLogItemParts = 4;        // up to 2^4 warps share an item of a short queue
constexpr uint32_t kLaneItems = 8;           // items a lane writes alone
constexpr uint32_t kLocalEdges = 512;        // frontier edges block 0 handles alone
constexpr uint32_t kGroupEdges = 16384;      // frontier edges the first kGroupBlocks blocks handle
constexpr unsigned kLogGroupBlocks = 4, kGroupBlocks = 1u << kLogGroupBlocks;
constexpr uint32_t kGroupItems = 4096;       // items per block of the group (more end the stretch)
constexpr uint32_t kPullMinEdges = 8192;     // a push with fewer frontier edges is never turned into a pull
constexpr uint32_t kLocalItems = 2048;       // items of a local level kept in shared memory (the rest spill)
constexpr uint32_t kLocalMaxLevels = 32768;  // levels per local or group stretch (the other blocks wait at a barrier)
constexpr int kPushUnroll = 4;               // edges per lane in flight in a push

// Item c of a list of d entries from s.
__device__ __forceinline__ uint2 list_item(uint32_t s, uint32_t d, uint32_t c) {
    return make_uint2(range_begin(s, kItemEdges, c), range_end(s, d, kItemEdges, c));
}

struct alignas(16) BfsSlot {
    unsigned long long edges;     // out-edges of the new frontier
    uint32_t discovered;          // vertices of the new frontier
    uint32_t items;               // its items (push)
    unsigned long long explored;  // stretch: out-edges of every vertex it labelled
    uint32_t levels;              // stretch: levels it advanced; items: whether some list made several
    uint32_t reached;             // stretch: vertices it labelled
};

// 16-byte accesses that are single and bypass L1: a value and its tag arrive
// together.
__device__ __forceinline__ void st_relaxed_16(uint4* p, const uint4& v) {
    asm volatile("{\n\t.reg .b128 q;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
                 "mov.b128 q, {a, b};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}
__device__ __forceinline__ uint4 ld_relaxed_16(const uint4* p) {
    uint4 v;
    asm volatile("{\n\t.reg .b128 q;\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.b128 q, [%4];\n\tmov.b128 {a, b}, q;\n\t"
                 "mov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

// Device memory of a search besides the graph-sized arrays, zeroed before it.
struct BfsSearchState {
    GridBarrier bar;
    GridBarrier group_bar;
    BfsSlot slot[3];
    uint4 entry[2][kGroupBlocks];  // the group's barrier: items, vertices, edges, phase of every block
    uint32_t overflow;             // the group's items beyond the blocks' segments (they end a stretch)
    uint32_t reached;
    int32_t level;
    uint32_t failed;
};

struct BfsSearch {
    const uint32_t* offsets;
    const uint32_t* targets;
    const uint32_t* active;  // list form of the pull
    uint32_t V, E, n_active, source;
    int symmetric;
    int32_t* dist;
    uint32_t* visited;
    uint32_t* bitmaps;  // three of bitmap_words each
    uint32_t bitmap_words;
    uint2* queue0;
    uint2* queue1;
    uint4* segments;  // the group's items: [2][kGroupBlocks][kGroupItems] (start, end, phase, epoch)
    uint32_t epoch;   // of this search among those of its segments, never 0
    BfsSearchState* st;
};

struct BfsLocal {
    uint32_t found, edges, items;
};

struct BfsShared {
    uint2 items[2][kLocalItems];
    unsigned long long edges[kSearchThreads / 32];
    uint32_t found[kSearchThreads / 32];
    BfsSlot slot;
    BfsLocal local[3];  // rotating like the slots: one block barrier per level
    uint32_t counts[kGroupBlocks];  // items of every block's segment
    BfsLocal all;                   // the group's counts of a level
    uint32_t over, ok;
};

__device__ __forceinline__ uint32_t* search_bitmap(const BfsSearch& a, uint32_t i) {
    return a.bitmaps + static_cast<size_t>(i) * a.bitmap_words;
}
__device__ __forceinline__ uint2* search_queue(const BfsSearch& a, uint32_t i) { return i ? a.queue1 : a.queue0; }

// Expands the q items of the frontier with the warps warp, warp + nwarps, ...
// of the blocks at work; new items go to the slot's `items` onwards of g_out. A warp
// takes consecutive items, whose lists are often neighbours in memory, but with
// `spread` items that are far apart: the items of a long list are consecutive, and
// 32 of them were one warp's while the others waited (a directed CSR of 4 hubs and
// 600,000 leaves: 700 of the level's 740 us).
__device__ __forceinline__ void push_items(const BfsSearch& a, const uint2* g_in, uint32_t q, bool spread, uint2* g_out,
                                           BfsSlot* slot, int32_t next_level, uint32_t warp, uint32_t nwarps,
                                           Tally& tally) {
    const unsigned lane = lane_id();
    uint32_t* const count = &slot->items;
    // Up to 32 items per warp at a time; with fewer items than warps, up to
    // 2^kLogItemParts warps share each.
    const uint32_t k = min(32u, max(1u, (q + nwarps - 1) / nwarps));
    const uint32_t parts = q ? min(1u << kLogItemParts, max(1u, nwarps / q)) : 1u;
    const uint32_t part = warp % parts;
    const uint32_t turns = range_count(q, k);
    for (uint32_t turn = warp / parts; turn < turns; turn += nwarps / parts) {
        const uint64_t i = spread ? turn + static_cast<uint64_t>(lane) * turns : static_cast<uint64_t>(turn) * k + lane;
        uint2 it = make_uint2(0u, 0u);
        if (lane < k && i < q) {
            it = __ldcg(g_in + i);
            if (parts > 1) {
                take_piece(it.x, it.y, part, (it.y - it.x + parts - 1) / parts);
            }
        }
        const uint32_t len = it.y - it.x;
        const uint32_t inc = warp_inclusive_scan(len);
        const uint32_t total = __shfl_sync(kFullMask, inc, 31);
        const uint32_t shift = it.x - (inc - len);  // entry of edge e of this item = shift + e
        for (uint32_t e0 = 0; e0 < total; e0 += 32 * kPushUnroll) {
            uint32_t v[kPushUnroll], ls[kPushUnroll], deg[kPushUnroll];
            bool found[kPushUnroll];
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) {
                const uint32_t e = e0 + u * 32 + lane;
                // The item of edge e: the number of items that end at or before it.
                uint32_t j = 0;
                if (k > 1) {
#pragma unroll
                    for (uint32_t step = 16; step > 0; step >>= 1)
                        if (__shfl_sync(kFullMask, inc, j + step - 1) <= e) j += step;
                }
                const uint32_t at = __shfl_sync(kFullMask, shift, j) + e;
                found[u] = e < total;
                v[u] = ld_nc_if(found[u], a.targets + at, 0u);
            }
            uint32_t word[kPushUnroll];
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) {
                word[u] = ld_cg_if(found[u], a.visited + (v[u] >> 5), 0xFFFFFFFFu);
            }
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) found[u] = !((word[u] >> (v[u] & 31)) & 1u);
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u)
                word[u] = atomic_or_if(found[u], a.visited + (v[u] >> 5), 1u << (v[u] & 31), 0xFFFFFFFFu);
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) found[u] = !((word[u] >> (v[u] & 31)) & 1u);
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) {
                ls[u] = ld_nc_if(found[u], a.offsets + v[u], 0u);
                deg[u] = ld_nc_if(found[u], a.offsets + v[u] + 1, 0u);
            }
            uint32_t mine = 0;
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) {
                deg[u] = found[u] ? deg[u] - ls[u] : 0u;
                if (found[u]) {
                    a.dist[v[u]] = next_level;
                    tally.found += 1;
                    tally.edges += deg[u];
                }
                mine += range_count(deg[u], kItemEdges);
            }
            const uint32_t upto = warp_inclusive_scan(mine);
            const uint32_t all = __shfl_sync(kFullMask, upto, 31);
            if (all == 0) continue;
            bool several = false;
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) several = several || deg[u] > kItemEdges;
            if (several) slot->levels = 1;
            uint32_t pos = 0;
            if (lane == 0) pos = atomicAdd(count, all);
            pos = __shfl_sync(kFullMask, pos, 0) + upto - mine;
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u) {
                const uint32_t n = range_count(deg[u], kItemEdges);
                if (n <= kLaneItems)
                    for (uint32_t c = 0; c < n; ++c) g_out[pos + c] = list_item(ls[u], deg[u], c);
                // Longer lists: the warp writes their items together.
                unsigned longs = __ballot_sync(kFullMask, n > kLaneItems);
                while (longs) {
                    const int l = __ffs(longs) - 1;
                    longs &= longs - 1;
                    const uint32_t s = __shfl_sync(kFullMask, ls[u], l), d = __shfl_sync(kFullMask, deg[u], l);
                    const uint32_t p = __shfl_sync(kFullMask, pos, l);
                    for (uint32_t c = lane; c < range_count(d, kItemEdges); c += 32) g_out[p + c] = list_item(s, d, c);
                }
                pos += n;
            }
        }
    }
}

// A stretch's level over the n items that read(i) gives, by 2^log_warps warps
// of which this is number `index`. Items are spread over as many lanes as there
// are: a warp takes k of them with 32 / k lanes each, and with fewer items
// than warps several warps share one (a warp whose 32 lanes issue scattered
// atomics waits about 9 cycles per lane for them, so few lanes per warp
// shorten the level's chain). put(at, s, e) stores item `at`
// of the new ones, numbered by the counter `count` in shared memory; when the
// warp's numbers pass `room`, spill(lo, hi) is called by all lanes for the numbers
// [lo, hi) past it, before their put().
constexpr uint32_t kLocalSolo = 8;  // edges per lane of an item before the whole warp takes it
constexpr int kStretchUnroll = 2;
constexpr uint32_t kLogBlockWarps = 5;
static_assert(kSearchThreads / 32 == 1 << kLogBlockWarps, "warps per block of a stretch");

template <class Read, class Spill, class Put>
__device__ __forceinline__ void stretch_items(const BfsSearch& a, uint32_t n, uint32_t index, uint32_t log_warps,
                                              int32_t next_level, uint32_t* count, uint32_t room, BfsLocal* c,
                                              Read read, Spill spill, Put put) {
    const unsigned lane = lane_id();
    uint32_t found_n = 0, found_m = 0;  // found_m: out-edges of a level's new vertices, below E < 2^32
    // Labels up to kPushUnroll edges of the list entries at, at + stride, ...
    // (all 32 lanes call it).
    auto expand = [&](uint32_t at, uint32_t end, uint32_t stride) {
        constexpr int kPushUnroll = kStretchUnroll;
        uint32_t v[kPushUnroll], ls[kPushUnroll], deg[kPushUnroll];
        bool ok[kPushUnroll];
#pragma unroll
        for (int u = 0; u < kPushUnroll; ++u) {
            ok[u] = at < end && end - at > u * stride;
            v[u] = ld_nc_if(ok[u], a.targets + at + u * stride, 0u);
        }
#pragma unroll
        for (int u = 0; u < kPushUnroll; ++u) {
            ls[u] = ld_nc_if(ok[u], a.offsets + v[u], 0u);
            deg[u] = ld_nc_if(ok[u], a.offsets + v[u] + 1, 0u);
        }
        uint32_t word[kPushUnroll];
#pragma unroll
        for (int u = 0; u < kPushUnroll; ++u)
            word[u] = atomic_or_if(ok[u], a.visited + (v[u] >> 5), 1u << (v[u] & 31), 0xFFFFFFFFu);
#pragma unroll
        for (int u = 0; u < kPushUnroll; ++u) ok[u] = !((word[u] >> (v[u] & 31)) & 1u);
        uint32_t mine = 0;
#pragma unroll
        for (int u = 0; u < kPushUnroll; ++u) {
            deg[u] = ok[u] ? deg[u] - ls[u] : 0u;
            if (ok[u]) {
                a.dist[v[u]] = next_level;
                found_n += 1;
                found_m += deg[u];
            }
            mine += range_count(deg[u], kItemEdges);
        }
        if (__ballot_sync(kFullMask, mine) == 0) return;
        const uint32_t upto = warp_inclusive_scan(mine);
        uint32_t pos = 0;
        if (lane == 31) pos = atomicAdd(count, upto);
        const uint32_t lo = __shfl_sync(kFullMask, pos, 31), hi = lo + __shfl_sync(kFullMask, upto, 31);
        if (hi > room) spill(max(lo, room), hi);
        pos = lo + upto - mine;
        bool one = true;  // at most one item per vertex
#pragma unroll
        for (int u = 0; u < kPushUnroll; ++u) one = one && deg[u] <= kItemEdges;
        if (__all_sync(kFullMask, one)) {
#pragma unroll
            for (int u = 0; u < kPushUnroll; ++u)
                if (deg[u]) put(pos++, ls[u], ls[u] + deg[u]);
            return;
        }
#pragma unroll
        for (int u = 0; u < kPushUnroll; ++u) {
            const uint32_t n = range_count(deg[u], kItemEdges);
            if (n <= kLaneItems)
                for (uint32_t k = 0; k < n; ++k) {
                    const uint2 it = list_item(ls[u], deg[u], k);
                    put(pos + k, it.x, it.y);
                }
            unsigned longs = __ballot_sync(kFullMask, n > kLaneItems);
            while (longs) {
                const int l = __ffs(longs) - 1;
                longs &= longs - 1;
                const uint32_t s = __shfl_sync(kFullMask, ls[u], l), d = __shfl_sync(kFullMask, deg[u], l);
                const uint32_t p = __shfl_sync(kFullMask, pos, l);
                for (uint32_t k = lane; k < range_count(d, kItemEdges); k += 32) {
                    const uint2 it = list_item(s, d, k);
                    put(p + k, it.x, it.y);
                }
            }
            pos += n;
        }
    };
    // Powers of two throughout: a division is a chain of some twenty instructions.
    const uint32_t warps = 1u << log_warps;
    const uint32_t k = min(32u, max(1u, (n + warps - 1) >> log_warps));
    const uint32_t log_parts = n == 0 || n > warps ? 0u : min(kLogItemParts, log_warps - (32 - __clz(n - 1)) % 32);
    const uint32_t log_lanes = k <= 1 ? 5u : __clz(k - 1) - 27u;  // 32 >> ceil(log2 k) lanes per item
    const uint32_t lanes = 1u << log_lanes;
    const uint32_t mine = lane & (lanes - 1), slot = lane >> log_lanes, part = index & ((1u << log_parts) - 1);
    for (uint32_t base = (index >> log_parts) * k; base < n; base += (warps >> log_parts) * k) {
        uint2 it = make_uint2(0u, 0u);
        if (slot < k && base + slot < n) {
            it = read(base + slot);
            if (log_parts) {
                take_piece(it.x, it.y, part, ((it.y - it.x) >> log_parts) + 1);
            }
        }
        const uint32_t len = it.y - it.x;
        const bool together = lanes < 32 && len > kLocalSolo * lanes;  // by the whole warp, after the others
        const uint32_t end = together ? it.x : it.y;
        const uint32_t longest = __reduce_max_sync(kFullMask, end - it.x);
        for (uint32_t o = 0; o < longest; o += lanes * kStretchUnroll) {
            expand(entry_or_end(it.x, end, min(o, end - it.x), mine), end, lanes);
        }
        unsigned longs = __ballot_sync(kFullMask, together && mine == 0);
        while (longs) {
            const int l = __ffs(longs) - 1;
            longs &= longs - 1;
            const uint32_t s = __shfl_sync(kFullMask, it.x, l), e = __shfl_sync(kFullMask, it.y, l);
            walk_entries(s, e, 32 * kStretchUnroll, [&](uint32_t b) { expand(entry_or_end(s, e, b, lane), e, 32); });
        }
    }
    found_n = __reduce_add_sync(kFullMask, found_n);
    found_m = __reduce_add_sync(kFullMask, found_m);
    if (lane == 0 && found_n) {
        atomicAdd(&c->found, found_n);
        atomicAdd(&c->edges, found_m);
    }
}

// Block 0 alone: item i of the frontier from s_in below kLocalItems and
// `shared`, else from g_in; new items to s_out below kLocalItems, else g_out.
__device__ __forceinline__ void local_level(const BfsSearch& a, const uint2* g_in, const uint2* s_in, bool shared,
                                            uint32_t q, uint2* g_out, uint2* s_out, BfsLocal* c, int32_t next_level) {
    stretch_items(
        a, q, threadIdx.x >> 5, kLogBlockWarps, next_level, &c->items, kLocalItems, c,
        [&](uint32_t i) { return shared && i < kLocalItems ? s_in[i] : __ldcg(g_in + i); },
        [](uint32_t, uint32_t) {},
        [&](uint32_t p, uint32_t s, uint32_t e) {
            if (p < kLocalItems) s_out[p] = make_uint2(s, e);
            else g_out[p] = make_uint2(s, e);
        });
}

// The group: block b's new items go to its segment of `out` (and, past
// kGroupItems, to g_out at positions from the shared counter `overflow`).
// Warp w of block b reads segment (b + w) % group, so every segment is read by
// warps of every block, whichever block filled it. An item carries the phase and
// the search that wrote it; a reader that comes before the item is there polls
// it, so the group's barrier needs no memory fence (a release waits about a
// microsecond for the level's scattered stores). What a reader may find instead
// of the item is an older one of the same segments, whose tag differs: the
// segments are cleared when they are allocated (the pool hands out memory in
// which another graph's searches left their items, whose tags repeat), the
// searches on them are numbered and so are a search's phases.
__device__ __forceinline__ void group_level(const BfsSearch& a, const uint2* queue, const uint4* in,
                                            const uint32_t* counts, bool first, uint32_t q, unsigned log_group, uint4* out,
                                            uint2* g_out, uint32_t phase, BfsLocal* c, int32_t next_level) {
    const uint32_t w = threadIdx.x >> 5;
    const uint32_t seg = (blockIdx.x + w) & ((1u << log_group) - 1);
    uint32_t shift = 0;  // g_out position of a spilled item less its number
    // The first level's items are one list in the queue. The warps that share
    // a segment: one of every block per `group` warps.
    stretch_items(
        a, first ? q : counts[seg], first ? (w << log_group) + blockIdx.x : w,
        first ? kLogBlockWarps + log_group : kLogBlockWarps, next_level,
        &c->items, kGroupItems, c,
        [&](uint32_t i) {
            if (first) return __ldcg(queue + i);
            const uint4* p = in + static_cast<size_t>(seg) * kGroupItems + i;
            uint4 v = ld_relaxed_16(p);
            for (unsigned k = 0; (v.z != phase - 1 || v.w != a.epoch) && k < kGridSpinLimit; ++k) {
                if ((k & 1023u) == 1023u && ld_relaxed(&a.st->bar.failed)) break;  // given up elsewhere
                v = ld_relaxed_16(p);
            }
            if (v.z != phase - 1 || v.w != a.epoch) {
                atomicExch(&a.st->bar.failed, 1u);
                return make_uint2(0u, 0u);
            }
            return make_uint2(v.x, v.y);
        },
        [&](uint32_t lo, uint32_t hi) {
            uint32_t at = 0;
            if (lane_id() == 0) at = atomicAdd(&a.st->overflow, hi - lo);
            shift = __shfl_sync(kFullMask, at, 0) - lo;
        },
        [&](uint32_t p, uint32_t s, uint32_t e) {
            if (p < kGroupItems) st_relaxed_16(out + static_cast<size_t>(blockIdx.x) * kGroupItems + p,
                                               make_uint4(s, e, phase, a.epoch));
            else g_out[shift + p] = make_uint2(s, e);
        });
}

// The group's barrier: every block posts its counts with the phase number in
// one 16-byte store, and the first warp of every block polls all of them (one
// lane each): no atomics, and the counts arrive with the last poll. It orders
// nothing else: inside a stretch the blocks share the visited bitmap (atomics)
// and tagged items only. Entries alternate by phase parity: a block posts
// phase p + 2 only after barrier p + 1, when everyone has read phase p.
// False: gave up (see grid_barrier).
__device__ __forceinline__ bool group_barrier(BfsSearchState* st, unsigned group, uint32_t phase, const BfsLocal& mine,
                                              BfsShared& sh) {
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned lane = lane_id();
        uint4* entry = st->entry[phase & 1];
        if (lane == 0) st_relaxed_16(entry + blockIdx.x, make_uint4(mine.items, mine.found, mine.edges, phase));
        bool ok = true;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (lane < group) {
            v = ld_relaxed_16(entry + lane);
            for (unsigned i = 0; v.w != phase; ++i) {
                if (i >= kGridSpinLimit || ((i & 1023u) == 1023u && ld_relaxed(&st->bar.failed))) {
                    atomicExch(&st->bar.failed, 1u);
                    ok = false;
                    break;
                }
                v = ld_relaxed_16(entry + lane);
            }
        }
        ok = __all_sync(kFullMask, ok);
        if (lane < group) sh.counts[lane] = v.x;
        const uint32_t items = __reduce_add_sync(kFullMask, v.x), found = __reduce_add_sync(kFullMask, v.y);
        const uint32_t edges = __reduce_add_sync(kFullMask, v.z);  // below E < 2^32
        const uint32_t over = __reduce_add_sync(kFullMask, v.x > kGroupItems ? v.x - kGroupItems : 0u);
        if (lane == 0) {
            sh.all = BfsLocal{found, edges, items};
            sh.over = over;
            sh.ok = ok ? 1u : 0u;
        }
    }
    __syncthreads();
    return sh.ok != 0;
}

// Whether one of the sector's eight entries targets[at .. at + 7] that lie in
// [s, e) is in the frontier (`at` a multiple of 8; the arrays are padded so
// that the last sector can be read whole). Two probes at a time, then four:
// lanes probe scattered words, so a probe costs the SM's L1 a tag lookup per
// lane, and in a wide frontier one of the first entries is usually a parent.
__device__ __forceinline__ bool probe_sector(uint32_t at, uint32_t s, uint32_t e, const uint32_t (&t)[8],
                                             const uint32_t* frontier) {
    uint32_t w[8];
    auto probe = [&](int i) { w[i] = ld_if(at + i >= s && at + i < e, frontier + (t[i] >> 5), 0u) >> (t[i] & 31); };
    probe(0), probe(1);
    if ((w[0] | w[1]) & 1u) return true;
    probe(2), probe(3);
    if ((w[2] | w[3]) & 1u) return true;
    probe(4), probe(5), probe(6), probe(7);
    return (w[4] | w[5] | w[6] | w[7]) & 1u;
}

// Pull level: a tile of 32 vertices per warp at a time. A lane reads
// its list in whole 32-byte sectors (8 entries, 8 frontier probes in flight),
// up to kSoloSectors of them; the lists still open after that are walked by
// the warp, 128 entries per step.
constexpr uint32_t kSoloSectors = 4;

template <bool kList>
__device__ __forceinline__ void pull_level(const BfsSearch& a, const uint32_t* frontier, uint32_t* next_frontier,
                                           int32_t next_level, uint32_t warp, uint32_t nwarps, Tally& tally) {
    const unsigned lane = lane_id();
    const uint64_t tiles = kList ? ceil_div_u64(a.n_active, 32) : ceil_div_u64(a.V, 32);
    uint32_t nv, ns, ne, nvis;
    // The next tile's vertices, visited words and list bounds are loaded while
    // the current one is probed.
    auto fetch = [&](uint64_t t) {
        nv = 0;
        ns = 0;
        ne = 0;
        nvis = 0xFFFFFFFFu;
        const uint64_t i = t * 32 + lane;
        if (i < (kList ? a.n_active : a.V)) {
            nv = kList ? __ldg(a.active + i) : static_cast<uint32_t>(i);
            nvis = a.visited[nv >> 5];
            ns = __ldg(a.offsets + nv);
            ne = __ldg(a.offsets + nv + 1);
        }
    };
    fetch(warp);
    for (uint64_t tile = warp; tile < tiles; tile += nwarps) {
        const uint32_t v = nv, s = ns, vis = nvis;
        uint32_t e = ne, t[8];
        if ((vis >> (v & 31)) & 1u) e = s;
        if (e > s) ld_stream8(a.targets + (s & ~7u), t);
        fetch(tile + nwarps);
        bool found = e > s && probe_sector(s & ~7u, s, e, t, frontier);
        // Rounded up in 64 bits: lists may end within a sector of 2^32.
        uint64_t at = (static_cast<uint64_t>(s) & ~7ull) + 8;
        for (uint32_t k = 1; k < kSoloSectors && at < e && !found; ++k, at += 8) {
            ld_stream8(a.targets + at, t);
            found = probe_sector(static_cast<uint32_t>(at), s, e, t, frontier);
        }
        unsigned pending = __ballot_sync(kFullMask, !found && at < e);
        while (pending) {
            const int p = __ffs(pending) - 1;
            pending &= pending - 1;
            const uint64_t ps = __shfl_sync(kFullMask, static_cast<uint32_t>(at), p);
            const uint64_t pe = __shfl_sync(kFullMask, e, p);
            bool hit = false;
            for (uint64_t b = ps; b < pe && !hit; b += 128) {
                const uint64_t j = b + 4 * lane;
                uint32_t h = 0;
                if (j < pe) {
                    const uint4 z = ld_stream4(reinterpret_cast<const uint4*>(a.targets + j));
                    const uint32_t h0 = ld_if(true, frontier + (z.x >> 5), 0u);
                    const uint32_t h1 = ld_if(j + 1 < pe, frontier + (z.y >> 5), 0u);
                    const uint32_t h2 = ld_if(j + 2 < pe, frontier + (z.z >> 5), 0u);
                    const uint32_t h3 = ld_if(j + 3 < pe, frontier + (z.w >> 5), 0u);
                    h = (h0 >> (z.x & 31)) | (h1 >> (z.y & 31)) | (h2 >> (z.z & 31)) | (h3 >> (z.w & 31));
                }
                hit = __any_sync(kFullMask, h & 1u);
            }
            if (static_cast<int>(lane) == p) found = hit;
        }
        if (found) {
            a.dist[v] = next_level;
            tally.found += 1;
            tally.edges += e - s;
        }
        if (kList) {
            // The tile's vertices ascend, so they share a few words: one
            // pair of atomics per word.
            if (__any_sync(kFullMask, found)) {
                const unsigned peers = __match_any_sync(kFullMask, v >> 5);
                const uint32_t bits = __reduce_or_sync(peers, found ? 1u << (v & 31) : 0u);
                if (bits && lane == static_cast<unsigned>(__ffs(peers) - 1)) {
                    atomicOr(next_frontier + (v >> 5), bits);
                    atomicOr(a.visited + (v >> 5), bits);
                }
            }
        } else {
            const unsigned mask = __ballot_sync(kFullMask, found);
            if (lane == 0) {
                next_frontier[tile] = mask;
                if (mask) a.visited[tile] = vis | mask;
            }
        }
    }
}

// The block's tallies into the level's slot, one atomic pair per block.
__device__ __forceinline__ void flush_block_tally(const Tally& tally, BfsShared& sh, BfsSlot* slot) {
    const uint32_t found = warp_sum(tally.found);
    const unsigned long long edges = warp_sum(tally.edges);
    const unsigned warp = threadIdx.x >> 5;
    if (lane_id() == 0) {
        sh.found[warp] = found;
        sh.edges[warp] = edges;
    }
    __syncthreads();
    if (warp == 0) {
        const unsigned lane = lane_id();
        const uint32_t f = warp_sum(lane < kSearchThreads / 32 ? sh.found[lane] : 0u);
        const unsigned long long m = warp_sum(lane < kSearchThreads / 32 ? sh.edges[lane] : 0ull);
        if (lane == 0 && f) {
            atomicAdd(&slot->discovered, f);
            atomicAdd(&slot->edges, m);
        }
    }
}

__device__ __forceinline__ void fetch_slot(const BfsSlot* slot, BfsSlot* to) {
    const uint4* p = reinterpret_cast<const uint4*>(slot);
    const uint4 x = __ldcg(p), y = __ldcg(p + 1);
    reinterpret_cast<uint4*>(to)[0] = x;
    reinterpret_cast<uint4*>(to)[1] = y;
}

template <bool kList>
__global__ void __launch_bounds__(kSearchThreads, kSearchCtasPerSm) bfs_search_kernel(const BfsSearch a) {
    __shared__ BfsShared sh;
    const unsigned lane = lane_id();
    const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t nthreads = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    // Warps of a block are spread over the grid's work (consecutive warps of
    // the numbering sit on different SMs), so a frontier of few items is not
    // left to one SM.
    const uint32_t nwarps = static_cast<uint32_t>(nthreads >> 5);
    const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t words = (a.V >> 5) + ((a.V & 31) ? 1u : 0u);
    unsigned barriers = 0;

    for (uint64_t i = tid; i * 4 < a.V; i += nthreads) {
        int4 d = make_int4(-1, -1, -1, -1);
        if (i == a.source >> 2) {
            const uint32_t c = a.source & 3;
            d = make_int4(c == 0 ? 0 : -1, c == 1 ? 0 : -1, c == 2 ? 0 : -1, c == 3 ? 0 : -1);
        }
        reinterpret_cast<int4*>(a.dist)[i] = d;
    }
    for (uint64_t i = tid; i < words; i += nthreads) {
        a.visited[i] = i == a.source >> 5 ? 1u << (a.source & 31) : 0u;
        if (kList) {
            search_bitmap(a, 0)[i] = 0;
            search_bitmap(a, 1)[i] = 0;
            search_bitmap(a, 2)[i] = 0;
        }
    }
    const uint32_t s0 = __ldg(a.offsets + a.source), d0 = __ldg(a.offsets + a.source + 1) - s0;
    uint32_t items = range_count(d0, kItemEdges);
    if (blockIdx.x == 0)
        for (uint32_t c = threadIdx.x; c < items; c += blockDim.x) a.queue0[c] = list_item(s0, d0, c);
    if (!grid_barrier(&a.st->bar, barriers)) {
        a.st->failed = 1;
        return;
    }

    unsigned long long m = d0, unexplored = a.E - d0;  // frontier edges, edges of unlabelled vertices
    uint32_t n = 1, reached = 1, cur = 0, bm = 0, phase = 0, group_phase = 0;
    int32_t level = 0;
    bool bottom_up = false, failed = false, spread = true;
    // Ends a phase: barrier, the phase's slot into shared memory.
    auto end_phase = [&]() -> bool {
        BfsSlot* slot = a.st->slot + phase % 3;
        const bool ok = grid_barrier(&a.st->bar, gridDim.x, barriers, [&] { fetch_slot(slot, &sh.slot); });
        ++phase;
        if (tid == 0) a.st->slot[(phase + 1) % 3] = BfsSlot{};
        if (!ok) a.st->failed = 1;
        return ok;
    };
    while (m > 0) {
        // A search labels each vertex once, so it ends within V levels with
        // at most V vertices reached; anything else can only be a fault.
        if (static_cast<uint32_t>(level) >= a.V || reached > a.V) {
            failed = true;
            break;
        }
        BfsSlot* slot = a.st->slot + phase % 3;
        // A small frontier is cheaper to push by the group than to pull (which
        // visits every vertex), whatever is left to explore.
        const bool pull = bfs_fixed_variant(a.symmetric != 0, bottom_up, n, m, unexplored, a.V) == kPull &&
                          (bottom_up || m > kPullMinEdges);
        Tally tally;
        bool local = false;
        if (pull) {
            if (!bottom_up) {  // the frontier bitmap from the distances
                uint32_t* bitmap = search_bitmap(a, bm);
                uint32_t* next = search_bitmap(a, (bm + 1) % 3);
                for (uint64_t w0 = static_cast<uint64_t>(warp) * 8; w0 < words;
                     w0 += static_cast<uint64_t>(nwarps) * 8) {
                    int32_t d[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const uint64_t v = (w0 + q) * 32 + lane;
                        d[q] = v < a.V ? a.dist[v] : -1;
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const unsigned mask = __ballot_sync(kFullMask, d[q] == level);
                        if (lane == 0 && w0 + q < words) {
                            bitmap[w0 + q] = mask;
                            if (kList) next[w0 + q] = 0;
                        }
                    }
                }
                if (!end_phase()) return;
                slot = a.st->slot + phase % 3;
            }
            if (kList) {  // the bitmap the next pull fills
                uint32_t* clear = search_bitmap(a, (bm + 2) % 3);
                for (uint64_t i = tid; i < words; i += nthreads) clear[i] = 0;
            }
            pull_level<kList>(a, search_bitmap(a, bm), search_bitmap(a, (bm + 1) % 3), level + 1, warp, nwarps, tally);
            flush_block_tally(tally, sh, slot);
        } else {
            if (bottom_up) {  // items of the frontier from its bitmap
                for (uint64_t w0 = static_cast<uint64_t>(warp) * 32; w0 < words;
                     w0 += static_cast<uint64_t>(nwarps) * 32) {
                    const uint32_t bits = w0 + lane < words ? search_bitmap(a, bm)[w0 + lane] : 0u;
                    // Each lane takes its word's vertices one by one.
                    for (uint32_t left = bits; __any_sync(kFullMask, left != 0); left &= left - 1) {
                        uint32_t s = 0, d = 0;
                        if (left) {
                            const uint32_t v = static_cast<uint32_t>((w0 + lane) * 32 + __ffs(left) - 1);
                            s = __ldg(a.offsets + v);
                            d = __ldg(a.offsets + v + 1) - s;
                        }
                        const uint32_t mine = range_count(d, kItemEdges);
                        if (mine > 1) slot->levels = 1;
                        const uint32_t upto = warp_inclusive_scan(mine);
                        uint32_t at = 0;
                        if (lane == 31 && upto) at = atomicAdd(&slot->items, upto);
                        at = __shfl_sync(kFullMask, at, 31) + upto - mine;
                        for (uint32_t c = 0; c < mine; ++c) search_queue(a, cur)[at + c] = list_item(s, d, c);
                    }
                }
                if (!end_phase()) return;
                items = sh.slot.items;
                spread = sh.slot.levels != 0;
                slot = a.st->slot + phase % 3;
            }
            local = m <= kGroupEdges;
            if (!local) {
                push_items(a, search_queue(a, cur), items, spread, search_queue(a, cur ^ 1), slot, level + 1, warp, nwarps,
                           tally);
                flush_block_tally(tally, sh, slot);
            } else {
                // A stretch of levels by block 0 or by the group, until the
                // frontier outgrows them or the search ends; the others wait.
                const bool alone = m <= kLocalEdges;
                const unsigned log_group = alone ? 0u : min(kLogGroupBlocks, 31 - __clz(gridDim.x));
                const unsigned group = 1u << log_group;
                if (blockIdx.x < group) {
                    uint32_t lq = items, lcur = cur, steps = 0, lreached = 0, ln = n;
                    unsigned long long lm = m, lexplored = 0;
                    if (threadIdx.x < 3) sh.local[threadIdx.x] = BfsLocal{};
                    __syncthreads();
                    while (true) {
                        const int32_t next_level = level + 1 + static_cast<int32_t>(steps);
                        BfsLocal* c = sh.local + steps % 3;
                        uint32_t found;
                        if (alone) {
                            // The frontier is in sh.items[steps & 1] (in the queue before the first level).
                            local_level(a, search_queue(a, lcur), sh.items[steps & 1], steps > 0, lq,
                                        search_queue(a, lcur ^ 1), sh.items[(steps & 1) ^ 1], c, next_level);
                            __syncthreads();
                            const BfsLocal r = *c;
                            found = r.found;
                            lm = r.edges;
                            if (found) lq = r.items;
                        } else {
                            // The frontier is in segments[steps & 1] (in the queue before the first level).
                            constexpr size_t kHalf = static_cast<size_t>(kGroupBlocks) * kGroupItems;
                            ++group_phase;
                            group_level(a, search_queue(a, lcur), a.segments + (steps & 1) * kHalf, sh.counts,
                                        steps == 0, lq, log_group, a.segments + ((steps & 1) ^ 1) * kHalf,
                                        search_queue(a, lcur ^ 1), group_phase, c, next_level);
                            if (!group_barrier(a.st, group, group_phase, *c, sh)) {
                                a.st->failed = 1;
                                return;
                            }
                            found = sh.all.found;
                            lm = sh.all.edges;
                            if (found) lq = sh.all.items;
                        }
                        // Slot (steps + 2) % 3 was read a level ago.
                        if (threadIdx.x == 0) sh.local[(steps + 2) % 3] = BfsLocal{};
                        if (found == 0) break;
                        steps += 1;
                        lreached += found;
                        lexplored += lm;
                        ln = found;
                        lcur ^= 1u;
                        if (lm == 0 || lm > (alone ? kLocalEdges : kGroupEdges) || steps >= kLocalMaxLevels) break;
                        // A frontier that has shrunk far enough is block 0's
                        // again; one that has outgrown a segment, everyone's.
                        if (!alone && (lm <= kLocalEdges / 2 || sh.over > 0)) break;
                    }
                    if (alone && steps > 0)
                        for (uint32_t i = threadIdx.x; i < min(lq, kLocalItems); i += blockDim.x)
                            search_queue(a, lcur)[i] = sh.items[steps & 1][i];
                    if (!alone && steps > 0) {
                        // The segments into the queue, after what overflowed.
                        uint32_t at = sh.over;
                        for (unsigned b = 0; b < blockIdx.x; ++b) at += min(sh.counts[b], kGroupItems);
                        const uint32_t mine = min(sh.counts[blockIdx.x], kGroupItems);
                        const uint4* from = a.segments + ((steps & 1) * kGroupBlocks + blockIdx.x) *
                                                             static_cast<size_t>(kGroupItems);
                        for (uint32_t i = threadIdx.x; i < mine; i += blockDim.x)
                            search_queue(a, lcur)[at + i] = make_uint2(__ldcg(from + i).x, __ldcg(from + i).y);
                    }
                    if (tid == 0) {
                        a.st->overflow = 0;
                        slot->edges = lm;
                        slot->explored = lexplored;
                        slot->discovered = ln;
                        slot->items = lq;
                        slot->levels = steps;
                        slot->reached = lreached;
                    }
                }
            }
        }
        if (!end_phase()) return;
        const BfsSlot r = sh.slot;
        if (local) {
            level += static_cast<int32_t>(r.levels);
            reached += r.reached;
            unexplored -= r.explored;
            cur ^= r.levels & 1u;
            spread = true;  // not known
        } else {
            spread = r.levels != 0;
            if (r.discovered == 0) break;  // the step labelled nothing: level and reached stay
            level += 1;
            reached += r.discovered;
            unexplored -= r.edges;
            if (pull) bm = (bm + 1) % 3;
            else cur ^= 1u;
        }
        n = r.discovered;
        m = r.edges;
        items = r.items;
        bottom_up = pull;
    }
    if (tid == 0) {
        a.st->reached = reached;
        a.st->level = level;
        if (failed) a.st->failed = 1;
    }
}

// ---------------------------------------------------------------- device-driven level loop (learned schedule)
//
// The host-driven loop reads the level counters back after every step (one
// copy and one synchronisation per level). The device-driven loop runs a
// whole search as one CUDA graph: a WHILE node whose body is a one-warp
// decide kernel followed by a SWITCH node over the three step variants. The
// decide kernel folds the last step's counters into BfsDevState exactly as
// the host's `advance` does, ends the loop where the host loop stops (empty
// frontier, or a step that labelled nothing), picks the next variant (the
// alpha/beta rule, or the learned schedule with its margin), and sets the
// SWITCH value; each step kernel reads its frontier size, level and queue
// parity from the state. The grids are fixed when the graph is captured and
// the kernels stride over what the state holds.

__global__ void bfs_loop_init_kernel(const uint32_t* __restrict__ offsets, uint32_t source,
                                     int32_t* __restrict__ dist, uint32_t* __restrict__ visited,
                                     uint32_t* __restrict__ queue0, BfsCounters* __restrict__ ctr,
                                     BfsDevState* __restrict__ st) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    dist[source] = 0;
    visited[source >> 5] |= 1u << (source & 31);
    const uint32_t deg = offsets[source + 1] - offsets[source];
    queue0[0] = source;
    BfsCounters c{};
    c.discovered = 1;
    c.queued = deg > 0 ? 1u : 0u;
    c.edges = deg;
    *ctr = c;
    BfsDevState s{};
    s.first = 1;
    s.variant = kSchedOut;
    *st = s;
}

__global__ void bfs_loop_decide_kernel(const __nv_bfloat16* __restrict__ w, BfsCounters* __restrict__ ctr,
                                       BfsDevState* __restrict__ st, DegreeStats stats, unsigned long long num_edges,
                                       uint32_t V, unsigned valid_mask, cudaGraphConditionalHandle h_loop,
                                       cudaGraphConditionalHandle h_step) {
    const BfsCounters c = *ctr;
    BfsDevState s = *st;
    bool stop = false;
    if (s.first) {
        s.first = 0;
        s.unexplored = num_edges - c.edges;
        s.reached = 1;
        s.level = 0;
    } else if (c.discovered == 0) {
        stop = true;  // the step labelled nothing: level and reached stay
    } else {
        s.level += 1;
        s.reached += c.discovered;
        s.unexplored -= c.edges;
        s.cur ^= 1u;
        s.bitmap_valid = s.variant == kPull ? 1u : 0u;
    }
    if (!stop) {
        s.frontier_n = c.discovered;
        s.frontier_q = c.queued;
        s.frontier_m = c.edges;
        stop = s.frontier_q == 0;
    }
    // A search labels each vertex once, so it ends within V levels with at
    // most V vertices reached and at most V queued; state past these bounds
    // can only come from a fault, and it ends the loop with the error flag
    // set instead of looping or indexing past the queues.
    if (!stop && (static_cast<uint64_t>(s.level) >= V || s.reached > V || s.frontier_q > V)) {
        stop = true;
        s.failed = 1;
    }
    int variant = kSchedOut;
    if (!stop) {
        variant = bfs_fixed_variant((valid_mask >> kPull) & 1u, s.bitmap_valid != 0, s.frontier_n, s.frontier_m,
                                    s.unexplored, V);
        if (w) {
            float f[kSchedIn];
            bfs_features(f, static_cast<float>(s.frontier_n), static_cast<float>(s.frontier_m),
                         static_cast<float>(s.unexplored), s.level, stats, s.bitmap_valid != 0,
                         static_cast<float>(s.reached));
            float out[kSchedOut];
            sched_forward_warp(w, f, out);
            const int pick = sched_pick_over(out, valid_mask, variant);
            if (pick >= 0) variant = pick;
        }
    }
    __syncwarp();
    if (lane_id() == 0) {
        s.variant = variant;
        *st = s;
        *ctr = BfsCounters{};
        cudaGraphSetConditional(h_step, static_cast<unsigned>(variant));
        cudaGraphSetConditional(h_loop, stop ? 0u : 1u);
    }
}

__global__ void __launch_bounds__(kTdThreads) bfs_topdown_warp_loop_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, uint32_t* queue0, uint32_t* queue1,
    int32_t* __restrict__ dist, uint32_t* __restrict__ visited, BfsCounters* __restrict__ ctr,
    const BfsDevState* __restrict__ st) {
    const uint32_t cur = st->cur;
    topdown_warp_body(offsets, targets, cur ? queue1 : queue0, st->frontier_q, dist, visited, cur ? queue0 : queue1,
                      ctr, st->level + 1);
}

// Also sets the IF node that picks the scan: three kernels above
// kScanOneLaunchMax frontier vertices, one below.
__global__ void bfs_queue_degrees_loop_kernel(const uint32_t* __restrict__ offsets, const uint32_t* queue0,
                                              const uint32_t* queue1, const BfsDevState* __restrict__ st,
                                              uint32_t* __restrict__ deg, int set_big,
                                              cudaGraphConditionalHandle h_big) {
    const uint32_t* queue = st->cur ? queue1 : queue0;
    const uint32_t n = st->frontier_q;
    if (set_big && blockIdx.x == 0 && threadIdx.x == 0)
        cudaGraphSetConditional(h_big, n > kScanOneLaunchMax ? 1u : 0u);
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t u = queue[i];
        deg[i] = offsets[u + 1] - offsets[u];
    }
}

// Balanced top-down over the scanned frontier degrees: blocks stride over the
// kTdTile-edge tiles of the frontier.
__global__ void __launch_bounds__(kTdThreads) bfs_topdown_loop_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, uint32_t* queue0, uint32_t* queue1,
    const uint32_t* __restrict__ qscan, int32_t* __restrict__ dist, uint32_t* __restrict__ visited,
    BfsCounters* __restrict__ ctr, const BfsDevState* __restrict__ st) {
    const uint32_t cur = st->cur, qsize = st->frontier_q;
    const int32_t next_level = st->level + 1;
    const uint32_t total = qscan[qsize];
    const uint32_t* queue = cur ? queue1 : queue0;
    uint32_t* next_queue = cur ? queue0 : queue1;
    Tally tally;
    const uint64_t tiles = ceil_div_u64(total, kTdTile);
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        topdown_tile(offsets, targets, queue, qsize, qscan, total, t * kTdTile, dist, visited, next_queue, ctr,
                     next_level, tally);
        __syncthreads();  // the tile's shared arrays are reused by the next tile
    }
    flush_tally(tally, ctr);
}

// Before a pull that follows a push: the frontier bitmap from the queue.
__global__ void bfs_bitmap_clear_loop_kernel(uint32_t* bitmap0, uint32_t* bitmap1, uint64_t words,
                                             const BfsDevState* __restrict__ st) {
    if (st->bitmap_valid) return;
    uint32_t* bitmap = st->cur ? bitmap1 : bitmap0;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < words;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        bitmap[i] = 0;
}

__global__ void bfs_queue_to_bitmap_loop_kernel(const uint32_t* queue0, const uint32_t* queue1, uint32_t* bitmap0,
                                                uint32_t* bitmap1, const BfsDevState* __restrict__ st) {
    if (st->bitmap_valid) return;
    const uint32_t* queue = st->cur ? queue1 : queue0;
    uint32_t* bitmap = st->cur ? bitmap1 : bitmap0;
    const uint32_t n = st->frontier_q;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t u = queue[i];
        atomicOr(bitmap + (u >> 5), 1u << (u & 31));
    }
}

template <bool kList>  // one instantiation per pull form, as bfs_bottomup_kernel
__global__ void __launch_bounds__(kBuThreads) bfs_bottomup_loop_kernel(
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ targets, uint32_t V,
    const uint32_t* __restrict__ active, uint32_t n_active, uint32_t* bitmap0, uint32_t* bitmap1,
    uint32_t* __restrict__ visited, int32_t* __restrict__ dist, uint32_t* queue0, uint32_t* queue1,
    BfsCounters* __restrict__ ctr, const BfsDevState* __restrict__ st) {
    const uint32_t cur = st->cur;
    if (kList)
        bottomup_list_body(offsets, targets, active, n_active, cur ? bitmap1 : bitmap0, cur ? bitmap0 : bitmap1,
                           visited, dist, cur ? queue0 : queue1, ctr, st->level + 1);
    else
        bottomup_body(offsets, targets, V, cur ? bitmap1 : bitmap0, cur ? bitmap0 : bitmap1, visited, dist,
                      cur ? queue0 : queue1, ctr, st->level + 1);
}

// The list form of the pull sets only found bits: clear the bitmap it fills.
__global__ void bfs_next_bitmap_clear_loop_kernel(uint32_t* bitmap0, uint32_t* bitmap1, uint64_t words,
                                                  const BfsDevState* __restrict__ st) {
    uint32_t* bitmap = st->cur ? bitmap0 : bitmap1;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < words;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        bitmap[i] = 0;
}

// ---------------------------------------------------------------- host

// The vertices with at least one entry, ascending (flags, scan, scatter).
__global__ void bfs_has_edges_kernel(const uint32_t* __restrict__ offsets, uint32_t V, uint32_t* __restrict__ flags) {
    for (uint64_t v = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
         v += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        flags[v] = offsets[v + 1] > offsets[v] ? 1u : 0u;
}

__global__ void bfs_active_scatter_kernel(const uint32_t* __restrict__ offsets, uint32_t V,
                                          const uint32_t* __restrict__ pos, uint32_t* __restrict__ active) {
    for (uint64_t v = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; v < V;
         v += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        if (offsets[v + 1] > offsets[v]) active[pos[v]] = static_cast<uint32_t>(v);
}

// No item of these segments has a tag that a search looks for (see group_level).
static Error clear_segments(DeviceImpl& dev, BfsWork& w) {
    GCU_CUDA(cudaMemsetAsync(w.search_segments.ptr, 0, sizeof(uint4) * w.search_segments.count, dev.stream), "memset");
    return ok();
}

static Error ensure_work(GraphImpl& g) {
    if (g.bfs_work) return ok();
    DeviceImpl& dev = *g.dev;
    auto w = std::unique_ptr<BfsWork, void (*)(BfsWork*)>(new BfsWork, destroy_bfs_work);
    const uint64_t V = g.num_nodes, words = ceil_div_u64(V, 32);
    GCU_TRY(w->dist.allocate(dev, V));
    GCU_TRY(w->visited.allocate(dev, words));
    // Bottom-up steps read in-neighbours; they equal the CSR lists only when
    // the CSR is symmetric (checked once per graph).
    bool sym = false;
    GCU_TRY(graph_symmetry(g, &sym));
    w->symmetric = sym ? 1 : 0;
    if (sym && V > 0) {
        DeviceBuffer<uint32_t> pos;  // flags, then positions
        GCU_TRY(pos.allocate(dev, V + 1));
        const unsigned grid = static_cast<unsigned>(
            std::min<uint64_t>(ceil_div_u64(V, 256), static_cast<uint64_t>(dev.sm_count) * 16));
        GCU_LAUNCH(dev, "bfs_has_edges", bfs_has_edges_kernel, grid, 256, 0, g.offsets.ptr, static_cast<uint32_t>(V),
                   pos.ptr);
        GCU_TRY(exclusive_scan_u32(dev, pos.ptr, pos.ptr, V));
        uint32_t n = 0;
        GCU_CUDA(cudaMemcpyAsync(&n, pos.ptr + V, sizeof(n), cudaMemcpyDeviceToHost, dev.stream), "copy");
        GCU_TRY(dev.sync());
        w->n_active = n;
        w->pull_list = V - n >= V / kBuListFraction;
        if (w->pull_list) {
            GCU_TRY(w->active.allocate(dev, std::max<uint32_t>(n, 1)));
            GCU_LAUNCH(dev, "bfs_active_scatter", bfs_active_scatter_kernel, grid, 256, 0, g.offsets.ptr,
                       static_cast<uint32_t>(V), pos.ptr, w->active.ptr);
        }
    }
    g.bfs_work = w.release();
    return ok();
}

// What the one-launch search works in, and what the levels by themselves do: a
// program that runs one form does not hold the other's (up to 24 bytes per vertex and
// 20; 36 with both).
static Error ensure_search(GraphImpl& g, BfsWork& w) {
    if (w.search_ready) return ok();
    DeviceImpl& dev = *g.dev;
    const uint64_t V = g.num_nodes;
    GCU_TRY(w.search_bitmaps.allocate(dev, 3 * ceil_div_u64(V, 32)));
    // At most one item per labelled vertex plus one per kItemEdges entries.
    for (auto& q : w.items) GCU_TRY(q.allocate(dev, V + g.num_edges / kItemEdges + 1));
    GCU_TRY(w.search_segments.allocate(dev, 2 * static_cast<size_t>(kGroupBlocks) * kGroupItems));
    GCU_TRY(clear_segments(dev, w));
    GCU_TRY(w.search.allocate(dev, 1));
    w.search_ready = true;
    return ok();
}

static Error ensure_levels(GraphImpl& g, BfsWork& w) {
    if (w.levels_ready) return ok();
    DeviceImpl& dev = *g.dev;
    const uint64_t V = g.num_nodes;
    for (auto& b : w.bitmap) GCU_TRY(b.allocate(dev, ceil_div_u64(V, 32)));
    for (auto& q : w.queue) GCU_TRY(q.allocate(dev, V));
    GCU_TRY(w.degree_scan.allocate(dev, V + 1));
    GCU_TRY(w.counters.allocate(dev, 1));
    w.levels_ready = true;
    return ok();
}

namespace {

// Where a level-synchronous run stands between two steps.
struct BfsState {
    uint32_t frontier_n = 0;    // vertices labelled by the last step
    uint32_t frontier_q = 0;    // of those, queued (out-degree > 0)
    uint64_t frontier_m = 0;    // their out-edges
    uint64_t unexplored = 0;    // out-edges of vertices not labelled yet
    uint32_t reached = 0;
    int32_t level = 0;          // level of the frontier
    int cur = 0;                // queue[cur] / bitmap[cur] hold the frontier
    bool bottom_up = false;     // the last step was a pull
    bool bitmap_valid = false;  // bitmap[cur] holds the frontier
};

int fixed_rule(const BfsState& st, bool symmetric, uint32_t V) {
    return bfs_fixed_variant(symmetric, st.bottom_up, st.frontier_n, st.frontier_m, st.unexplored, V);
}

unsigned valid_variants(bool symmetric) {
    return (1u << kPushWarp) | (1u << kPushBalanced) | (symmetric ? (1u << kPull) : 0u);
}

// Launches one step of `variant` from the frontier in st (counters reset).
Error launch_step(GraphImpl& g, BfsWork& w, int variant, const BfsState& st) {
    DeviceImpl& dev = *g.dev;
    const uint32_t V = g.num_nodes;
    const uint64_t words = ceil_div_u64(V, 32);
    const unsigned grid_cap = static_cast<unsigned>(dev.sm_count) * 16;
    const int cur = st.cur, nxt = cur ^ 1;
    GCU_CUDA(cudaMemsetAsync(w.counters.ptr, 0, sizeof(BfsCounters), dev.stream), "memset");
    if (variant == kPull) {
        if (!st.bitmap_valid) {
            GCU_CUDA(cudaMemsetAsync(w.bitmap[cur].ptr, 0, sizeof(uint32_t) * words, dev.stream), "memset");
            unsigned blocks = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(st.frontier_q, 256), grid_cap));
            GCU_LAUNCH(dev, "bfs_queue_to_bitmap", bfs_queue_to_bitmap_kernel, blocks, 256, 0, w.queue[cur].ptr,
                       st.frontier_q, w.bitmap[cur].ptr);
        }
        const uint64_t lanes = w.pull_list ? w.n_active : words * 32;
        if (w.pull_list)
            GCU_CUDA(cudaMemsetAsync(w.bitmap[nxt].ptr, 0, sizeof(uint32_t) * words, dev.stream), "memset");
        unsigned blocks = static_cast<unsigned>(
            std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(lanes, kBuThreads), grid_cap)));
        const auto bottomup = w.pull_list ? bfs_bottomup_kernel<true> : bfs_bottomup_kernel<false>;
        GCU_LAUNCH(dev, "bfs_bottomup", bottomup, blocks, kBuThreads, 0, g.offsets.ptr, g.targets.ptr, V,
                   w.pull_list ? w.active.ptr : nullptr, w.n_active, w.bitmap[cur].ptr, w.bitmap[nxt].ptr, w.visited.ptr, w.dist.ptr,
                   w.queue[nxt].ptr, w.counters.ptr, st.level + 1);
    } else if (variant == kPushWarp) {
        unsigned blocks = static_cast<unsigned>(
            std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(st.frontier_q, kTdThreads / 32), grid_cap)));
        GCU_LAUNCH(dev, "bfs_topdown_warp", bfs_topdown_warp_kernel, blocks, kTdThreads, 0, g.offsets.ptr,
                   g.targets.ptr, w.queue[cur].ptr, st.frontier_q, w.dist.ptr, w.visited.ptr, w.queue[nxt].ptr,
                   w.counters.ptr, st.level + 1);
    } else {
        unsigned blocks = static_cast<unsigned>(std::min<uint64_t>(ceil_div_u64(st.frontier_q, 256), grid_cap));
        GCU_LAUNCH(dev, "bfs_queue_degrees", bfs_queue_degrees_kernel, blocks, 256, 0, g.offsets.ptr,
                   w.queue[cur].ptr, st.frontier_q, w.degree_scan.ptr);
        GCU_TRY(exclusive_scan_u32(dev, w.degree_scan.ptr, w.degree_scan.ptr, st.frontier_q));
        unsigned td_blocks = static_cast<unsigned>(std::max<uint64_t>(1, ceil_div_u64(st.frontier_m, kTdTile)));
        GCU_LAUNCH(dev, "bfs_topdown", bfs_topdown_kernel, td_blocks, kTdThreads, 0, g.offsets.ptr, g.targets.ptr,
                   w.queue[cur].ptr, st.frontier_q, w.degree_scan.ptr, w.dist.ptr, w.visited.ptr, w.queue[nxt].ptr,
                   w.counters.ptr, st.level + 1);
    }
    return ok();
}

// Resets the work buffers and labels the source; st describes level 0.
Error start_run(GraphImpl& g, BfsWork& w, uint32_t source) {
    DeviceImpl& dev = *g.dev;
    const uint64_t words = ceil_div_u64(g.num_nodes, 32);
    GCU_CUDA(cudaMemsetAsync(w.dist.ptr, 0xFF, sizeof(int32_t) * g.num_nodes, dev.stream), "memset");
    GCU_CUDA(cudaMemsetAsync(w.visited.ptr, 0, sizeof(uint32_t) * words, dev.stream), "memset");
    GCU_CUDA(cudaMemsetAsync(w.counters.ptr, 0, sizeof(BfsCounters), dev.stream), "memset");
    GCU_LAUNCH(dev, "bfs_init", bfs_init_kernel, 1, 32, 0, g.offsets.ptr, source, w.dist.ptr, w.visited.ptr,
               w.queue[0].ptr, w.counters.ptr);
    return ok();
}

Error read_counters(DeviceImpl& dev, BfsWork& w) {
    GCU_CUDA(cudaMemcpyAsync(&w.host_counters, w.counters.ptr, sizeof(BfsCounters), cudaMemcpyDeviceToHost, dev.stream),
             "copy");
    return dev.sync();
}

// Folds the counters of the step just run (or of the init) into st.
void advance(BfsState& st, const BfsCounters& c, bool first, int variant, uint64_t num_edges) {
    if (first) {
        st.unexplored = num_edges - c.edges;
        st.reached = 1;
        st.level = 0;
    } else {
        st.level += 1;
        st.reached += c.discovered;
        st.unexplored -= c.edges;
        st.cur ^= 1;
        st.bottom_up = variant == kPull;
        st.bitmap_valid = variant == kPull;
    }
    st.frontier_n = c.discovered;
    st.frontier_q = c.queued;
    st.frontier_m = c.edges;
}

// Captures the launches `f` makes on the device stream into `target` (a
// conditional node's body graph), after the node `after` when given.
template <class F>
Error capture_into(DeviceImpl& dev, cudaGraph_t target, F&& f, const cudaGraphNode_t* after = nullptr) {
    GCU_CUDA(cudaStreamBeginCaptureToGraph(dev.stream, target, after, nullptr, after ? 1 : 0,
                                           cudaStreamCaptureModeThreadLocal),
             "cudaStreamBeginCaptureToGraph");
    const Error e = f();
    cudaGraph_t captured = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(dev.stream, &captured);
    GCU_TRY(e);
    if (ce != cudaSuccess) return driver_error(ce, "cudaStreamEndCapture");
    return ok();
}

// The graph of a device-driven search: WHILE(loop) { decide; SWITCH(step) {
// push with a warp per vertex | balanced push | pull } }. Everything it reads
// lives in the BfsWork buffers and the graph's CSR; the source is labelled by
// bfs_loop_init_kernel before each launch.
Error build_loop_graph(GraphImpl& g, BfsWork& w) {
    DeviceImpl& dev = *g.dev;
    if (w.loop_exec) {
        cudaGraphExecDestroy(w.loop_exec);
        w.loop_exec = nullptr;
    }
    if (w.loop_graph) {
        cudaGraphDestroy(w.loop_graph);
        w.loop_graph = nullptr;
    }
    const uint32_t V = g.num_nodes;
    const uint64_t words = ceil_div_u64(V, 32);
    if (!w.loop_state.ptr) {
        GCU_TRY(w.loop_state.allocate(dev, 1));
        GCU_TRY(w.loop_scan_sums.allocate(dev, scan_device_n_tiles(V)));
    }
    const __nv_bfloat16* net = reinterpret_cast<const __nv_bfloat16*>(dev.schedule);
    DegreeStats stats;
    if (net) GCU_TRY(degree_stats(g, &stats));
    const bool sym = w.symmetric == 1;
    const unsigned valid = valid_variants(sym);
    BfsDevState* st = w.loop_state.ptr;
    const uint32_t* n_ptr = &st->frontier_q;
    const unsigned cap = static_cast<unsigned>(dev.sm_count) * 16;
    const unsigned vgrid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(V, 256), cap)));
    const unsigned bu_grid = static_cast<unsigned>(std::max<uint64_t>(
        1, std::min<uint64_t>(ceil_div_u64(w.pull_list ? w.n_active : words * 32, kBuThreads), cap)));
    const unsigned wgrid =
        static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(ceil_div_u64(V, kTdThreads / 32), cap)));
    const unsigned td_grid = static_cast<unsigned>(dev.sm_count) * 8;

    cudaGraph_t graph = nullptr;
    GCU_CUDA(cudaGraphCreate(&graph, 0), "cudaGraphCreate");
    struct Owner {
        cudaGraph_t g;
        ~Owner() {
            if (g) cudaGraphDestroy(g);
        }
    } owner{graph};
    cudaGraphConditionalHandle h_loop = 0, h_step = 0;
    GCU_CUDA(cudaGraphConditionalHandleCreate(&h_loop, graph, 1, cudaGraphCondAssignDefault),
             "cudaGraphConditionalHandleCreate");
    cudaGraphNodeParams wp = {};
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = h_loop;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    cudaGraphNode_t while_node = nullptr;
    GCU_CUDA(cudaGraphAddNode(&while_node, graph, nullptr, 0, &wp), "cudaGraphAddNode (while)");
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    GCU_CUDA(cudaGraphConditionalHandleCreate(&h_step, body, 0, 0), "cudaGraphConditionalHandleCreate");
    GCU_TRY(capture_into(dev, body, [&]() -> Error {
        GCU_LAUNCH(dev, "bfs_loop_decide", bfs_loop_decide_kernel, 1, 32, 0, net, w.counters.ptr, st, stats,
                   static_cast<unsigned long long>(g.num_edges), V, valid, h_loop, h_step);
        return ok();
    }));
    cudaGraphNode_t decide_node = nullptr;
    size_t nodes = 1;
    GCU_CUDA(cudaGraphGetNodes(body, &decide_node, &nodes), "cudaGraphGetNodes");
    if (nodes != 1) return kernel_error("BFS loop graph: unexpected body");
    cudaGraphNodeParams sp = {};
    sp.type = cudaGraphNodeTypeConditional;
    sp.conditional.handle = h_step;
    sp.conditional.type = cudaGraphCondTypeSwitch;
    sp.conditional.size = kSchedOut;
    cudaGraphNode_t switch_node = nullptr;
    GCU_CUDA(cudaGraphAddNode(&switch_node, body, &decide_node, 1, &sp), "cudaGraphAddNode (switch)");
    cudaGraph_t* branch = sp.conditional.phGraph_out;
    GCU_TRY(capture_into(dev, branch[kPushWarp], [&]() -> Error {
        GCU_LAUNCH(dev, "bfs_topdown_warp", bfs_topdown_warp_loop_kernel, wgrid, kTdThreads, 0, g.offsets.ptr,
                   g.targets.ptr, w.queue[0].ptr, w.queue[1].ptr, w.dist.ptr, w.visited.ptr, w.counters.ptr, st);
        return ok();
    }));
    // Balanced push: degrees (which set the scan's IF), IF(n > 8192) { three-kernel
    // scan } ELSE { one-kernel scan }, expand. Graphs of at most 8192
    // vertices only ever take the one-kernel scan: no IF node.
    cudaGraph_t balanced = branch[kPushBalanced];
    const bool big = V > kScanOneLaunchMax;
    cudaGraphConditionalHandle h_big = 0;
    if (big)
        GCU_CUDA(cudaGraphConditionalHandleCreate(&h_big, balanced, 0, 0), "cudaGraphConditionalHandleCreate");
    auto launch_expand = [&]() -> Error {
        GCU_LAUNCH(dev, "bfs_topdown", bfs_topdown_loop_kernel, td_grid, kTdThreads, 0, g.offsets.ptr, g.targets.ptr,
                   w.queue[0].ptr, w.queue[1].ptr, w.degree_scan.ptr, w.dist.ptr, w.visited.ptr, w.counters.ptr, st);
        return ok();
    };
    GCU_TRY(capture_into(dev, balanced, [&]() -> Error {
        GCU_LAUNCH(dev, "bfs_queue_degrees", bfs_queue_degrees_loop_kernel, vgrid, 256, 0, g.offsets.ptr,
                   w.queue[0].ptr, w.queue[1].ptr, st, w.degree_scan.ptr, big ? 1 : 0, h_big);
        if (big) return ok();
        GCU_TRY(exclusive_scan_u32_device_n(dev, w.degree_scan.ptr, w.degree_scan.ptr, n_ptr, V,
                                            w.loop_scan_sums.ptr, ScanLaunches::kOneTile));
        return launch_expand();
    }));
    if (big) {
        cudaGraphNode_t degrees_node = nullptr;
        nodes = 1;
        GCU_CUDA(cudaGraphGetNodes(balanced, &degrees_node, &nodes), "cudaGraphGetNodes");
        if (nodes != 1) return kernel_error("BFS loop graph: unexpected balanced branch");
        cudaGraphNodeParams ip = {};
        ip.type = cudaGraphNodeTypeConditional;
        ip.conditional.handle = h_big;
        ip.conditional.type = cudaGraphCondTypeIf;
        ip.conditional.size = 2;
        cudaGraphNode_t if_node = nullptr;
        GCU_CUDA(cudaGraphAddNode(&if_node, balanced, &degrees_node, 1, &ip), "cudaGraphAddNode (if)");
        GCU_TRY(capture_into(dev, ip.conditional.phGraph_out[0], [&]() -> Error {
            return exclusive_scan_u32_device_n(dev, w.degree_scan.ptr, w.degree_scan.ptr, n_ptr, V,
                                               w.loop_scan_sums.ptr, ScanLaunches::kMultiTile);
        }));
        GCU_TRY(capture_into(dev, ip.conditional.phGraph_out[1], [&]() -> Error {
            return exclusive_scan_u32_device_n(dev, w.degree_scan.ptr, w.degree_scan.ptr, n_ptr, V,
                                               w.loop_scan_sums.ptr, ScanLaunches::kOneTile);
        }));
        GCU_TRY(capture_into(dev, balanced, launch_expand, &if_node));
    }
    GCU_TRY(capture_into(dev, branch[kPull], [&]() -> Error {
        GCU_LAUNCH(dev, "bfs_bitmap_clear", bfs_bitmap_clear_loop_kernel, vgrid, 256, 0, w.bitmap[0].ptr,
                   w.bitmap[1].ptr, words, st);
        GCU_LAUNCH(dev, "bfs_queue_to_bitmap", bfs_queue_to_bitmap_loop_kernel, vgrid, 256, 0, w.queue[0].ptr,
                   w.queue[1].ptr, w.bitmap[0].ptr, w.bitmap[1].ptr, st);
        if (w.pull_list)
            GCU_LAUNCH(dev, "bfs_next_bitmap_clear", bfs_next_bitmap_clear_loop_kernel, vgrid, 256, 0,
                       w.bitmap[0].ptr, w.bitmap[1].ptr, words, st);
        const auto bottomup = w.pull_list ? bfs_bottomup_loop_kernel<true> : bfs_bottomup_loop_kernel<false>;
        GCU_LAUNCH(dev, "bfs_bottomup", bottomup, bu_grid, kBuThreads, 0, g.offsets.ptr,
                   g.targets.ptr, V, w.pull_list ? w.active.ptr : nullptr, w.n_active, w.bitmap[0].ptr, w.bitmap[1].ptr, w.visited.ptr,
                   w.dist.ptr, w.queue[0].ptr, w.queue[1].ptr, w.counters.ptr, st);
        return ok();
    }));
    cudaGraphExec_t exec = nullptr;
    GCU_CUDA(cudaGraphInstantiate(&exec, graph, 0), "cudaGraphInstantiate");
    w.loop_graph = graph;
    owner.g = nullptr;
    w.loop_exec = exec;
    w.loop_net = net;
    return ok();
}

// One search through the loop graph; the final state gives reachable and
// max_depth.
Error run_loop(GraphImpl& g, BfsWork& w, uint32_t source, BfsDevState* final_state) {
    DeviceImpl& dev = *g.dev;
    const uint64_t words = ceil_div_u64(g.num_nodes, 32);
    GCU_CUDA(cudaMemsetAsync(w.dist.ptr, 0xFF, sizeof(int32_t) * g.num_nodes, dev.stream), "memset");
    GCU_CUDA(cudaMemsetAsync(w.visited.ptr, 0, sizeof(uint32_t) * words, dev.stream), "memset");
    GCU_LAUNCH(dev, "bfs_init", bfs_loop_init_kernel, 1, 32, 0, g.offsets.ptr, source, w.dist.ptr, w.visited.ptr,
               w.queue[0].ptr, w.counters.ptr, w.loop_state.ptr);
    dev.launches.fetch_add(1, std::memory_order_relaxed);
    GCU_CUDA(cudaGraphLaunch(w.loop_exec, dev.stream), "cudaGraphLaunch");
    GCU_CUDA(cudaMemcpyAsync(&w.host_loop_state, w.loop_state.ptr, sizeof(BfsDevState), cudaMemcpyDeviceToHost,
                             dev.stream),
             "copy");
    GCU_TRY(dev.sync());
    *final_state = w.host_loop_state;
    return ok();
}

// Blocks of the one-launch search: all that are resident at once for a large
// graph, one per kSearchVertices vertices or kSearchEntries entries for a
// small one (fewer blocks meet faster at a barrier).
constexpr uint64_t kSearchVertices = 2048;
constexpr uint64_t kSearchEntries = 16384;

// One search as one cooperative launch.
Error run_search(GraphImpl& g, BfsWork& w, uint32_t source) {
    DeviceImpl& dev = *g.dev;
    const auto kernel = w.pull_list ? bfs_search_kernel<true> : bfs_search_kernel<false>;
    if (!w.search_grid) {
        int per_sm = 0;
        GCU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSearchThreads, 0), "occupancy");
        const uint64_t most = static_cast<uint64_t>(dev.sm_count) * std::max(1, std::min(per_sm, kSearchCtasPerSm));
        const uint64_t want = std::max<uint64_t>(
            {1, ceil_div_u64(g.num_nodes, kSearchVertices), ceil_div_u64(g.num_edges, kSearchEntries)});
        w.search_grid = static_cast<unsigned>(std::min(want, most));
    }
    BfsSearch a{};
    a.offsets = g.offsets.ptr;
    a.targets = g.targets.ptr;
    a.active = w.pull_list ? w.active.ptr : nullptr;
    a.V = g.num_nodes;
    a.E = g.num_edges;
    a.n_active = w.n_active;
    a.source = source;
    a.symmetric = w.symmetric == 1 ? 1 : 0;
    a.dist = w.dist.ptr;
    a.visited = w.visited.ptr;
    a.bitmaps = w.search_bitmaps.ptr;
    a.bitmap_words = static_cast<uint32_t>(ceil_div_u64(g.num_nodes, 32));
    a.queue0 = w.items[0].ptr;
    a.queue1 = w.items[1].ptr;
    a.segments = w.search_segments.ptr;
    if (++w.search_epoch == 0) {  // the numbers begin again
        GCU_TRY(clear_segments(dev, w));
        w.search_epoch = 1;
    }
    a.epoch = w.search_epoch;
    a.st = w.search.ptr;
    GCU_CUDA(cudaMemsetAsync(w.search.ptr, 0, sizeof(BfsSearchState), dev.stream), "memset");
    GCU_LAUNCH_COOP(dev, "bfs_search", kernel, w.search_grid, kSearchThreads, 0, a);
    GCU_CUDA(cudaMemcpyAsync(&w.host_search, &w.search.ptr->reached, sizeof(w.host_search), cudaMemcpyDeviceToHost,
                             dev.stream),
             "copy");
    return ok();
}

uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

}  // namespace

Error bfs(GraphImpl& g, uint32_t source, int32_t* host_distances, uint32_t* reachable, int32_t* max_depth) {
    DeviceImpl& dev = *g.dev;
    GCU_TRY(ensure_work(g));
    BfsWork& w = *g.bfs_work;
    const bool sym = w.symmetric == 1;
    const unsigned valid = valid_variants(sym);
    const __nv_bfloat16* net = reinterpret_cast<const __nv_bfloat16*>(dev.schedule);
    DegreeStats stats;
    if (net) GCU_TRY(degree_stats(g, &stats));

    if (dev.bfs_device_loop && !dev.kernel_timing && !net) {
        const Error ready = ensure_search(g, w);
        if (ready.ok()) {
            GCU_TRY(run_search(g, w, source));
            if (host_distances)
                GCU_TRY(copy_to_host(dev, host_distances, w.dist.ptr, sizeof(int32_t) * g.num_nodes));
            GCU_TRY(dev.sync());
            if (w.host_search.failed) return kernel_error("BFS stopped on an impossible state");
            *reachable = w.host_search.reached;
            *max_depth = w.host_search.level;
            return ok();
        }
        if (ready.status != GCU_ERR_OUT_OF_MEMORY) return ready;
        for (auto& q : w.items) q.reset();  // the levels need less
    }
    GCU_TRY(ensure_levels(g, w));
    if (dev.bfs_device_loop && !dev.kernel_timing && !w.loop_unavailable) {
        if (!w.loop_exec || w.loop_net != static_cast<const void*>(net)) {
            // A driver that cannot build the conditional graph leaves the
            // search to the host-driven loop below (same kernels, same result).
            if (!build_loop_graph(g, w).ok()) w.loop_unavailable = true;
        }
        if (w.loop_exec) {
            BfsDevState fin{};
            GCU_TRY(run_loop(g, w, source, &fin));
            if (fin.failed) return kernel_error("BFS level loop stopped on an impossible state");
            if (host_distances)
                GCU_TRY(copy_to_host(dev, host_distances, w.dist.ptr, sizeof(int32_t) * g.num_nodes));
            *reachable = fin.reached;
            *max_depth = fin.level;
            return ok();
        }
    }

    GCU_TRY(start_run(g, w, source));
    if (net)
        GCU_LAUNCH(dev, "bfs_decide", bfs_decide_kernel, 1, 32, 0, net, w.counters.ptr, stats,
                   static_cast<unsigned long long>(g.num_edges), 0u, 0, 0, valid, g.num_nodes, nullptr);
    GCU_TRY(read_counters(dev, w));
    BfsState st;
    advance(st, w.host_counters, true, 0, g.num_edges);
    while (st.frontier_q > 0) {
        int variant = fixed_rule(st, sym, g.num_nodes);
        if (net) {
            const int c = w.host_counters.choice;
            if (c >= 0 && ((valid >> c) & 1u)) variant = c;
        }
        GCU_TRY(launch_step(g, w, variant, st));
        if (net)
            GCU_LAUNCH(dev, "bfs_decide", bfs_decide_kernel, 1, 32, 0, net, w.counters.ptr, stats,
                       static_cast<unsigned long long>(st.unexplored), st.reached, st.level + 1,
                       variant == kPull ? 1 : 0, valid, g.num_nodes, nullptr);
        GCU_TRY(read_counters(dev, w));
        if (w.host_counters.discovered == 0) break;
        advance(st, w.host_counters, false, variant, g.num_edges);
    }
    if (host_distances) GCU_TRY(copy_to_host(dev, host_distances, w.dist.ptr, sizeof(int32_t) * g.num_nodes));
    *reachable = st.reached;
    *max_depth = st.level;
    return ok();
}

// Trace: at every level, each valid variant runs from the same frontier
// (visited bitmap and distances restored from a snapshot in between) and is
// timed with events on the stream; all must label the same vertices. The run
// then continues with the fixed rule's variant, or, for 3 levels in 10 chosen
// by explore_seed, a uniformly drawn valid one (so that the traces also hold
// states the fixed rule never reaches).
Error bfs_trace(GraphImpl& g, uint32_t source, uint64_t explore_seed, std::vector<BfsTraceLevel>* levels) {
    DeviceImpl& dev = *g.dev;
    GCU_TRY(ensure_work(g));
    BfsWork& w = *g.bfs_work;
    GCU_TRY(ensure_levels(g, w));
    const bool sym = w.symmetric == 1;
    const unsigned valid = valid_variants(sym);
    DegreeStats stats;
    GCU_TRY(degree_stats(g, &stats));
    const uint64_t V = g.num_nodes, words = ceil_div_u64(V, 32);
    DeviceBuffer<uint32_t> visited_snap;
    DeviceBuffer<int32_t> dist_snap;
    DeviceBuffer<BfsCounters> variant_ctr;
    DeviceBuffer<float> feats;
    GCU_TRY(visited_snap.allocate(dev, words));
    GCU_TRY(dist_snap.allocate(dev, V));
    GCU_TRY(variant_ctr.allocate(dev, kSchedOut));
    cudaEvent_t ev[2 * kSchedOut];
    for (auto& e : ev) GCU_CUDA(cudaEventCreate(&e), "cudaEventCreate");
    struct Events {
        cudaEvent_t* e;
        ~Events() {
            for (int i = 0; i < 2 * kSchedOut; ++i) cudaEventDestroy(e[i]);
        }
    } guard{ev};

    levels->clear();
    GCU_TRY(feats.allocate(dev, kSchedIn));
    GCU_TRY(start_run(g, w, source));
    GCU_LAUNCH(dev, "bfs_decide", bfs_decide_kernel, 1, 32, 0, nullptr, w.counters.ptr, stats,
               static_cast<unsigned long long>(g.num_edges), 0u, 0, 0, valid, g.num_nodes, feats.ptr);
    GCU_TRY(read_counters(dev, w));
    BfsState st;
    advance(st, w.host_counters, true, 0, g.num_edges);
    std::vector<float> host_feats(kSchedIn);
    GCU_CUDA(cudaMemcpy(host_feats.data(), feats.ptr, 4 * kSchedIn, cudaMemcpyDeviceToHost), "copy");
    while (st.frontier_q > 0) {
        BfsTraceLevel rec{};
        for (int k = 0; k < kSchedIn; ++k) rec.features[k] = host_feats[k];
        rec.valid = static_cast<uint8_t>(valid);
        const int fixed = fixed_rule(st, sym, g.num_nodes);
        rec.fixed_rule = static_cast<uint8_t>(fixed);
        int take = fixed;
        const uint64_t r = mix64(explore_seed * 0x9E3779B97F4A7C15ull + static_cast<uint64_t>(st.level) + 1);
        if (r % 10 < 3) {
            const int nvalid = __builtin_popcount(valid);
            int pick = static_cast<int>((r >> 32) % nvalid);
            for (int c = 0; c < kSchedOut; ++c)
                if ((valid >> c) & 1u) {
                    if (pick == 0) {
                        take = c;
                        break;
                    }
                    --pick;
                }
        }
        rec.taken = static_cast<uint8_t>(take);
        GCU_CUDA(cudaMemcpyAsync(visited_snap.ptr, w.visited.ptr, 4 * words, cudaMemcpyDeviceToDevice, dev.stream),
                 "copy");
        GCU_CUDA(cudaMemcpyAsync(dist_snap.ptr, w.dist.ptr, 4 * V, cudaMemcpyDeviceToDevice, dev.stream), "copy");
        for (int k = 0; k < kSchedOut; ++k) {
            const int c = (k + st.level) % kSchedOut;  // rotate which variant goes first
            if (!((valid >> c) & 1u)) continue;
            GCU_CUDA(cudaEventRecord(ev[2 * c], dev.stream), "cudaEventRecord");
            GCU_TRY(launch_step(g, w, c, st));
            GCU_CUDA(cudaEventRecord(ev[2 * c + 1], dev.stream), "cudaEventRecord");
            GCU_CUDA(cudaMemcpyAsync(variant_ctr.ptr + c, w.counters.ptr, sizeof(BfsCounters),
                                     cudaMemcpyDeviceToDevice, dev.stream),
                     "copy");
            GCU_CUDA(cudaMemcpyAsync(w.visited.ptr, visited_snap.ptr, 4 * words, cudaMemcpyDeviceToDevice, dev.stream),
                     "copy");
            GCU_CUDA(cudaMemcpyAsync(w.dist.ptr, dist_snap.ptr, 4 * V, cudaMemcpyDeviceToDevice, dev.stream), "copy");
        }
        GCU_TRY(launch_step(g, w, take, st));
        GCU_LAUNCH(dev, "bfs_decide", bfs_decide_kernel, 1, 32, 0, nullptr, w.counters.ptr, stats,
                   static_cast<unsigned long long>(st.unexplored), st.reached, st.level + 1, take == kPull ? 1 : 0,
                   valid, g.num_nodes, feats.ptr);
        BfsCounters vc[kSchedOut];
        GCU_CUDA(cudaMemcpyAsync(vc, variant_ctr.ptr, sizeof(vc), cudaMemcpyDeviceToHost, dev.stream), "copy");
        GCU_CUDA(cudaMemcpyAsync(host_feats.data(), feats.ptr, 4 * kSchedIn, cudaMemcpyDeviceToHost, dev.stream),
                 "copy");
        GCU_TRY(read_counters(dev, w));
        const BfsCounters c = w.host_counters;
        for (int v = 0; v < kSchedOut; ++v) {
            rec.times_us[v] = __builtin_nanf("");
            if (!((valid >> v) & 1u)) continue;
            if (vc[v].discovered != c.discovered || vc[v].queued != c.queued || vc[v].edges != c.edges)
                return kernel_error("BFS step variants disagree at level " + std::to_string(st.level));
            float ms = 0.f;
            GCU_CUDA(cudaEventElapsedTime(&ms, ev[2 * v], ev[2 * v + 1]), "cudaEventElapsedTime");
            rec.times_us[v] = 1000.f * ms;
        }
        levels->push_back(rec);
        if (c.discovered == 0) break;
        advance(st, c, false, take, g.num_edges);
    }
    return ok();
}

}  // namespace gcu

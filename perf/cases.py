"""Performance cases: the calls a program makes on grafeo_cuda, over their range of sizes.

Each case is one call (or one short sequence of calls) through the public Python
module on a graph whose structure comes from the case's seed. The families and
sizes are those of bench.py, the tests and the device generators: R-MAT with
(0.57, 0.19, 0.19) and 8 to 32 pairs per vertex, Erdos-Renyi G(n, m), the 2D
grid with dropped edges (long diameter), Watts-Strogatz, the directed R-MAT copy
with 3 % dangling vertices, and the packed batch of many small graphs. Graphs are
drawn here with torch, so that the inputs do not depend on the library's own
generators, and handed over as host CSR arrays.

listed(): the fixed cases. draw(rng): one more case of the same ranges.
prepare(case, seed): the inputs and handles a program holds before the call.
run(state): one pass. work(case): bytes and flops a pass cannot do without.
exact(case, seed): the floating-point outputs of run() in FP64, computed with
torch alone.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "grafeo-cuda_b200"))

DAMPING = 0.85
_device = None


def device():
    """The one GpuDevice a program keeps for its lifetime."""
    global _device
    if _device is None:
        import grafeo_cuda

        _device = grafeo_cuda.GpuDevice(0)
    return _device


# ---------------------------------------------------------------- cases


def listed():
    return [
        # One search on a small social graph, distances back: launch latency is the cost.
        {"name": "bfs_rmat14", "kind": "bfs", "family": "rmat", "nodes": 1 << 14, "degree": 16, "sources": 1},
        # Road-like graph: about two thousand levels with small frontiers, distances back.
        {"name": "bfs_grid_1024", "kind": "bfs", "family": "grid", "nodes": 1 << 20, "degree": 4, "sources": 1},
        # Graph500 style: searches from 16 vertices of a large graph, reach and depth of each.
        {"name": "bfs_rmat22_x16", "kind": "bfs", "family": "rmat", "nodes": 1 << 22, "degree": 16, "sources": 16},
        # The small benchmark configuration: 20 iterations, ranks back.
        {"name": "pagerank_rmat14", "kind": "pagerank", "family": "rmat", "nodes": 1 << 14, "degree": 16,
         "iterations": 20, "tolerance": 0.0, "directed": False, "seeds": 0},
        # Default arguments on a large graph without hubs.
        {"name": "pagerank_er22", "kind": "pagerank", "family": "er", "nodes": 1 << 22, "degree": 16,
         "iterations": 100, "tolerance": 1e-6, "directed": False, "seeds": 0},
        # The headline: directed, 3 % dangling, to an L1 change below 1e-7.
        {"name": "pagerank_directed_rmat24", "kind": "pagerank", "family": "rmat", "nodes": 1 << 24, "degree": 16,
         "iterations": 100, "tolerance": 1e-7, "directed": True, "seeds": 0},
        # Triangle counts of an ordinary and of a large graph.
        {"name": "triangles_rmat16", "kind": "triangles", "family": "rmat", "nodes": 1 << 16, "degree": 16},
        {"name": "triangles_rmat22", "kind": "triangles", "family": "rmat", "nodes": 1 << 22, "degree": 16},
        # A program that loads a graph and asks for its 4-truss (whole call: upload, support, peel, edges).
        {"name": "ktruss_rmat18", "kind": "ktruss", "family": "rmat", "nodes": 1 << 18, "degree": 16, "k": 4},
        # Truss decomposition of a resident graph: thousands of peeling rounds.
        {"name": "truss_rmat19", "kind": "truss", "family": "rmat", "nodes": 1 << 19, "degree": 16},
        # Many small graphs in one captured replay: triangles, 16-source BFS, personalised PageRank of each.
        {"name": "batch_256", "kind": "batch", "graphs": 256, "sources": 16, "seeds": 8, "iterations": 20},
        # An edge list in host memory to the ranks of its graph (whole call: build, plan, iterate).
        {"name": "edges_to_ranks_16m", "kind": "edges", "family": "rmat", "nodes": 1 << 20, "degree": 16,
         "iterations": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bfs", "bfs", "pagerank", "pagerank", "triangles", "triangles", "ktruss", "truss", "batch",
                       "edges"])
    degree = rng.randint(8, 24)
    if kind == "bfs":
        family = rng.choice(["rmat", "er", "grid", "ws"])
        if family == "grid":
            return {"kind": kind, "family": family, "nodes": _log_int(rng, 40, 1024) ** 2, "degree": 4, "sources": 1}
        if family == "ws":
            return {"kind": kind, "family": family, "nodes": _log_int(rng, 2000, 1 << 21), "degree": 10,
                    "sources": rng.choice([1, 4])}
        nodes = _log_int(rng, 1 << 10, 1 << 22)
        return {"kind": kind, "family": family, "nodes": nodes, "degree": min(degree, (1 << 26) // nodes),
                "sources": rng.choice([1, 4, 16])}
    if kind == "pagerank":
        nodes = _log_int(rng, 1 << 10, 1 << 23)
        fixed = rng.random() < 0.5
        return {"kind": kind, "family": rng.choice(["rmat", "rmat", "er", "ws"]), "nodes": nodes,
                "degree": min(degree, (1 << 27) // nodes), "iterations": rng.choice([10, 20, 50]) if fixed else 100,
                "tolerance": 0.0 if fixed else 1e-6, "directed": rng.random() < 0.4,
                "seeds": rng.choice([0, 0, 1, 8])}
    if kind == "triangles":
        nodes = _log_int(rng, 1 << 10, 1 << 22)
        return {"kind": kind, "family": rng.choice(["rmat", "rmat", "er", "ws"]), "nodes": nodes,
                "degree": min(degree, (1 << 26) // nodes)}
    if kind == "ktruss":
        nodes = _log_int(rng, 1 << 10, 1 << 18)
        return {"kind": kind, "family": rng.choice(["rmat", "er", "ws"]), "nodes": nodes,
                "degree": min(degree, (1 << 22) // nodes), "k": rng.randint(3, 6)}
    if kind == "truss":
        nodes = _log_int(rng, 1 << 10, 1 << 19)
        return {"kind": kind, "family": rng.choice(["rmat", "rmat", "ws"]), "nodes": nodes,
                "degree": min(degree, (1 << 23) // nodes)}
    if kind == "batch":
        return {"kind": kind, "graphs": _log_int(rng, 8, 256), "sources": rng.choice([1, 8, 16, 32]),
                "seeds": rng.choice([1, 8]), "iterations": 20}
    nodes = _log_int(rng, 1 << 10, 1 << 20)
    return {"kind": kind, "family": rng.choice(["rmat", "er"]), "nodes": nodes,
            "degree": min(degree, (1 << 24) // nodes), "iterations": 20}


# ---------------------------------------------------------------- inputs (torch on the GPU)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rmat_pairs(n, m, g):
    """m R-MAT pairs over n vertices: ids drawn over 2^ceil(log2 n), scaled down to n."""
    bits = max(1, math.ceil(math.log2(n)))
    s = torch.zeros(m, dtype=torch.int64, device="cuda")
    d = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(bits):
        u = torch.rand(m, device="cuda", generator=g)
        s.mul_(2).add_(u >= 0.76)
        d.mul_(2).add_(((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    if n != 1 << bits:
        s.mul_(n).bitwise_right_shift_(bits)
        d.mul_(n).bitwise_right_shift_(bits)
    return s, d


def _ws_pairs(n, k, g):
    half = max(1, k // 2)
    s = torch.arange(n, device="cuda").repeat_interleave(half)
    d = (s + torch.arange(1, half + 1, device="cuda").repeat(n)) % n
    far = torch.randint(0, n, (s.numel(),), device="cuda", generator=g)
    return s, torch.where(torch.rand(s.numel(), device="cuda", generator=g) < 0.1, far, d)


def _pairs(family, n, degree, g):
    if family == "rmat":
        return _rmat_pairs(n, n * degree, g)
    if family == "er":
        m = n * degree
        return (torch.randint(0, n, (m,), device="cuda", generator=g),
                torch.randint(0, n, (m,), device="cuda", generator=g))
    if family == "ws":
        return _ws_pairs(n, 10, g)
    side = math.isqrt(n)  # grid
    at = torch.arange(side * side, device="cuda").view(side, side)
    s = torch.cat([at[:, :-1].reshape(-1), at[:-1].reshape(-1)])
    d = torch.cat([at[:, 1:].reshape(-1), at[1:].reshape(-1)])
    keep = torch.rand(s.numel(), device="cuda", generator=g) >= 0.05
    return s[keep], d[keep]


def _keys(s, d, symmetric=True):
    """Sorted distinct (source << 32) | target keys without self-loops."""
    loop = s == d
    k = (s << 32) | d
    if symmetric:
        k = torch.cat([k[~loop], ((d << 32) | s)[~loop]])
    else:
        k = k[~loop]
    k = torch.sort(k).values
    if k.numel():
        first = torch.ones(k.numel(), dtype=torch.bool, device="cuda")
        torch.ne(k[1:], k[:-1], out=first[1:])
        k = k[first]
    return k


def _offsets(keys, n):
    rows = torch.arange(n + 1, device="cuda", dtype=torch.int64) << 32
    return torch.searchsorted(keys, rows)


def _counted_keys(case, seed):
    """A graph of exactly _counted_edges(case) edges: pairs are drawn until enough are distinct,
    then that many of them are kept at random."""
    n, want = case["nodes"], _counted_edges(case)
    g = _gen(seed)
    degree = case["degree"]
    while True:
        s, d = _pairs(case["family"], n, degree, g)
        once = _keys(torch.minimum(s, d), torch.maximum(s, d), symmetric=False)
        if once.numel() >= want:
            break
        degree = degree * 3 // 2
    kept = torch.randperm(once.numel(), device="cuda", generator=g)[:want]
    once = once[kept]
    return _keys(once >> 32, once & 0xFFFFFFFF), n


def _counted_edges(case):
    return int(0.85 * {"ws": 5}.get(case["family"], case["degree"]) * case["nodes"])


def _graph_keys(case, seed):
    """(keys, n) of the case's graph; a directed one loses the out-edges of 3 % of its vertices."""
    if case["kind"] == "truss":
        return _counted_keys(case, seed)
    n = case["nodes"]
    g = _gen(seed)
    s, d = _pairs(case["family"], n, case["degree"], g)
    keys = _keys(s, d)
    del s, d
    if case.get("directed"):
        live = torch.rand(n, device="cuda", generator=g) >= 0.03
        keys = keys[live[keys >> 32]]
    return keys, n


def _host(t):
    return t.to(torch.int32).cpu().numpy().view(np.uint32)


def _host_csr(keys, n):
    offsets = _host(_offsets(keys, n))
    targets = _host(keys & 0xFFFFFFFF)
    return offsets, targets


def _live_vertices(offsets, count, seed):
    """`count` vertices with edges, drawn from the seed."""
    live = np.nonzero(np.diff(offsets.astype(np.int64)))[0]
    return live[np.random.default_rng(seed).integers(0, len(live), size=count)].astype(np.uint32)


def _batch_keys(case, seed):
    """A union of R-MAT (scale 8..16, 8..32 pairs per vertex) and Watts-Strogatz
    (256..65536 vertices) graphs with equal odds: (keys, vertex_base). The sizes
    depend on the number of graphs alone, the edges on the seed."""
    rng = np.random.default_rng(case["graphs"])
    g = _gen(seed)
    base, parts = [0], []
    for _ in range(case["graphs"]):
        if rng.random() < 0.5:
            n = 1 << int(rng.integers(8, 17))
            s, d = _rmat_pairs(n, n * int(rng.integers(8, 33)), g)
        else:
            n = int(rng.integers(256, 65537))
            s, d = _ws_pairs(n, 10, g)
        parts.append((s + base[-1], d + base[-1]))
        base.append(base[-1] + n)
    keys = _keys(torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts]))
    return keys, np.array(base, dtype=np.uint32)


def _batch_vertices(offsets, base, count, seed):
    """[graphs, count] local ids of vertices with edges."""
    rng = np.random.default_rng(seed)
    degree = np.diff(offsets.astype(np.int64))
    out = np.zeros((len(base) - 1, count), dtype=np.uint32)
    for i in range(len(base) - 1):
        live = np.nonzero(degree[base[i]:base[i + 1]])[0]
        out[i] = live[rng.integers(0, len(live), size=count)]
    return out


def prepare(case, seed):
    import grafeo_cuda

    dev = device()
    state = {"case": case}
    if case["kind"] == "edges":
        s, d = _pairs(case["family"], case["nodes"], case["degree"], _gen(seed))
        state["edges"] = np.stack([_host(s), _host(d)], axis=1)
        return state
    if case["kind"] == "batch":
        keys, base = _batch_keys(case, seed)
        offsets, targets = _host_csr(keys, int(base[-1]))
        del keys
        torch.cuda.empty_cache()
        b = grafeo_cuda.GpuBatch.from_csr(base, offsets, targets, dev)
        b.set_bfs_sources(_batch_vertices(offsets, base, case["sources"], seed + 1), keep_distances=False)
        b.set_pagerank_seeds(_batch_vertices(offsets, base, case["seeds"], seed + 2), DAMPING, case["iterations"], 0.0)
        b.capture()
        state["batch"] = b
        return state
    keys, n = _graph_keys(case, seed)
    offsets, targets = _host_csr(keys, n)
    del keys
    torch.cuda.empty_cache()
    if case["kind"] == "ktruss":
        state["csr"] = (offsets, targets)
        # The program's own array for the edges: room for every edge of the graph.
        state["edges"] = np.zeros((case["nodes"] * case["degree"], 2), dtype=np.int32)
        return state
    state["graph"] = grafeo_cuda.GpuGraph.from_csr(offsets, targets, dev)
    if case["kind"] == "bfs":
        state["sources"] = [int(v) for v in _live_vertices(offsets, case["sources"], seed + 1)]
    if case["kind"] == "pagerank" and case["seeds"]:
        state["seeds"] = _live_vertices(offsets, case["seeds"], seed + 1)
    return state


# ---------------------------------------------------------------- one pass


def run(state):
    import grafeo_cuda

    case = state["case"]
    kind = case["kind"]
    if kind == "bfs":
        g = state["graph"]
        last = len(state["sources"]) - 1
        results = [g.bfs_array(s, copy_result=i == last) for i, s in enumerate(state["sources"])]
        return {"distances": results[-1]["distances"],
                "reachable": np.array([r["reachable"] for r in results], dtype=np.int64),
                "max_depth": np.array([r["max_depth"] for r in results], dtype=np.int64)}
    if kind == "pagerank":
        g = state["graph"]
        args = (DAMPING, case["iterations"], case["tolerance"])
        if "seeds" in state:
            r = g.personalized_pagerank(state["seeds"], *args, directed=case["directed"])
        elif case["directed"]:
            r = g.pagerank_directed(*args)
        else:
            r = g.pagerank_array(*args)
        return {"ranks": r["ranks"], "converged": r["converged"]}
    if kind == "triangles":
        return {"total": state["graph"].triangle_count()["total_triangles"]}
    if kind == "ktruss":
        g = grafeo_cuda.GpuGraph.from_csr(*state["csr"], device())
        r = g.k_truss_array(case["k"])
        m, edges = len(r["edges"]), state["edges"]
        edges[:m] = r["edges"]
        edges[m:] = 0
        return {"edges": edges, "count": m, "rounds": r["iterations"]}
    if kind == "truss":
        r = state["graph"].truss_decomposition()
        return {"trussness": r["trussness"].view(np.int32), "max": r["max_trussness"], "rounds": r["rounds"]}
    if kind == "batch":
        state["batch"].replay()
        r = state["batch"].results(distances=False)
        return {"triangles": r["total_triangles"].astype(np.int64), "reachable": r["reachable"].view(np.int32),
                "max_depth": r["max_depth"], "ranks": r["ranks"]}
    g = grafeo_cuda.GpuGraph.from_edge_pairs(state["edges"], case["nodes"], True, device())
    return {"ranks": g.pagerank_array(DAMPING, case["iterations"], 0.0)["ranks"], "num_edges": g.num_edges}


# ---------------------------------------------------------------- what a pass cannot do without


def _sweeps(case):
    """PageRank iterations: the given number, or about as many as an L1 change
    that shrinks by 0.65 a step needs to pass the tolerance."""
    if case.get("tolerance"):
        return min(case["iterations"], math.ceil(math.log(case["tolerance"]) / math.log(0.65)))
    return case["iterations"]


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n, e = 24000 * case["graphs"], 410000 * case["graphs"]
        # Triangles and BFS read the lists once each, every PageRank sweep once.
        return {"bytes": (2 + case["iterations"]) * (4 * e + 12 * n), "flops": 2 * case["iterations"] * e}
    n = case["nodes"]
    degree = {"ws": 5, "grid": 2}.get(case["family"], case["degree"])
    e = 2 * degree * n
    if kind == "bfs":
        return {"bytes": case["sources"] * (4 * e + 8 * n), "flops": 0}
    if kind == "pagerank":
        return {"bytes": _sweeps(case) * (4 * e + 12 * n), "flops": 2 * _sweeps(case) * e}
    if kind == "edges":
        # The pairs, the CSR written, then every sweep.
        return {"bytes": 4 * e + 4 * e + case["iterations"] * (4 * e + 12 * n), "flops": 2 * case["iterations"] * e}
    if kind == "triangles":
        return {"bytes": 4 * e + 4 * n, "flops": 0}
    if kind == "ktruss":
        return {"bytes": 8 * e + 4 * n, "flops": 0}  # lists in, kept pairs out
    e = 2 * _counted_edges(case)
    return {"bytes": 8 * e + 4 * n, "flops": 0}  # truss: lists in, trussness out


# ---------------------------------------------------------------- FP64


def _sweep_matrix(keys, n):
    """Pull matrix over the lists as a torch CSR matrix of ones, and the row lengths."""
    offsets = _offsets(keys, n)
    ones = torch.ones(keys.numel(), dtype=torch.float64, device="cuda")
    m = torch.sparse_csr_tensor(offsets.to(torch.int32), (keys & 0xFFFFFFFF).to(torch.int32), ones, size=(n, n))
    return m, (offsets[1:] - offsets[:-1]).double()


def _pagerank64(matrix, outdeg, group, sizes, tele, iterations, tolerance):
    """Power iteration r = (1 - d) p + d (A c + dangling p), started at 1 / n, per group of vertices."""
    d = float(np.float32(DAMPING))
    r = 1.0 / sizes[group]
    dangling_row = outdeg == 0
    inv = torch.where(dangling_row, torch.zeros_like(outdeg), 1.0 / outdeg.clamp(min=1.0))
    for _ in range(iterations):
        mass = torch.zeros_like(sizes).index_add_(0, group, torch.where(dangling_row, r, torch.zeros_like(r)))
        new = (1.0 - d) * tele + d * (matrix @ (r * inv) + mass[group] * tele)
        change = float((new - r).abs().sum())
        r = new
        if change < float(np.float32(tolerance)):
            break
    return r


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("pagerank", "edges", "batch"):
        return None
    if kind == "batch":
        keys, base = _batch_keys(case, seed)
        n = int(base[-1])
        sizes = np.diff(base.astype(np.int64))
        group = torch.from_numpy(np.repeat(np.arange(len(sizes)), sizes)).cuda()
        offsets = _host(_offsets(keys, n))
        seeds = _batch_vertices(offsets, base, case["seeds"], seed + 2).astype(np.int64) + base[:-1, None]
        tele = torch.zeros(n, dtype=torch.float64, device="cuda")
        tele.index_add_(0, torch.from_numpy(seeds.reshape(-1)).cuda(),
                        torch.full((seeds.size,), 1.0 / case["seeds"], dtype=torch.float64, device="cuda"))
        matrix, outdeg = _sweep_matrix(keys, n)
        ranks = _pagerank64(matrix, outdeg, group, torch.from_numpy(sizes).double().cuda(), tele,
                            case["iterations"], 0.0)
        return {"triangles": None, "reachable": None, "max_depth": None, "ranks": ranks}
    n = case["nodes"]
    if kind == "edges":
        keys = _keys_with_loops(case, seed)
    else:
        keys, n = _graph_keys(case, seed)
    group = torch.zeros(n, dtype=torch.int64, device="cuda")
    sizes = torch.tensor([float(n)], dtype=torch.float64, device="cuda")
    tele = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    if case.get("seeds"):
        seeds = torch.from_numpy(_live_vertices(_host(_offsets(keys, n)), case["seeds"], seed + 1).astype(np.int64))
        tele = torch.zeros(n, dtype=torch.float64, device="cuda")
        tele.index_add_(0, seeds.cuda(), torch.full((len(seeds),), 1.0 / len(seeds), dtype=torch.float64,
                                                    device="cuda"))
    matrix, outdeg = _sweep_matrix(keys, n)
    if case.get("directed"):
        keys = torch.sort(((keys & 0xFFFFFFFF) << 32) | (keys >> 32)).values
        matrix, _ = _sweep_matrix(keys, n)
    del keys
    torch.cuda.empty_cache()
    ranks = _pagerank64(matrix, outdeg, group, sizes, tele, case["iterations"], case.get("tolerance", 0.0))
    out = {"ranks": ranks}
    out["num_edges" if kind == "edges" else "converged"] = None
    return out


def _keys_with_loops(case, seed):
    """The edge-list case keeps self-loops (once), as from_edge_pairs does."""
    s, d = _pairs(case["family"], case["nodes"], case["degree"], _gen(seed))
    k = torch.sort(torch.cat([(s << 32) | d, (d << 32) | s])).values
    first = torch.ones(k.numel(), dtype=torch.bool, device="cuda")
    torch.ne(k[1:], k[:-1], out=first[1:])
    return k[first]

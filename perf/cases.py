"""What a user of this framework has it do, as cases that can be timed and compared.

Every case takes one graph, built from an edge list on the device, through one
public entry point: single-source BFS, batched BFS, SSSP, connected components,
betweenness centrality, triangle counting, graph construction, or a BFS / SSSP
loop written with the advance / filter operators.  Graphs are the kinds the
benchmark, the autotuner's training set and the tests use: RMAT (0.57, 0.19,
0.19, 0.05), uniform random, and 4-neighbour grids with or without random
long-range pairs.  Results are read where a program on the GPU would read them
(the instances' device arrays).

A case's fields: "kind" (the entry point), "graph" / "n" / "degree" (generated
pairs per vertex; of a grid, n = side * side) / "long_range" (pairs added to a
grid, as a share of its own) / "relabel" (vertex ids shuffled: RMAT's hubs
otherwise have the low ids) / "directed" / "weights", and the options of the
entry point.
"""
import ctypes
import math

import numpy as np
import torch

import sygraph_b200 as sg
from sygraph_b200 import _lib
from sygraph_b200._lib import call
from sygraph_b200.core import DeviceArray

A, B, C = 0.57, 0.19, 0.19
ALPHA, BETA = 15.0, 24.0  # single-source direction switch, as the benchmark sets it
ALPHA_BATCHED = 4.0
MAX_U32_WEIGHT = 64


# ------------------------------------------------------------------ the cases
def case(kind, graph, n, degree=16, *, long_range=0.0, relabel=False, directed=False, weights="f32", **options):
    return {"kind": kind, "graph": graph, "n": n, "degree": degree, "long_range": long_range, "relabel": relabel,
            "directed": directed, "weights": weights, **options}


def listed():
    return [
        # a query on a graph that fits a cache: launch latency and the chain of a few tiny levels
        {"name": "bfs_rmat10", **case("bfs", "rmat", 1 << 10, direction="hybrid")},
        # the benchmark's headline: one traversal of RMAT-22
        {"name": "bfs_rmat22", **case("bfs", "rmat", 1 << 22, direction="hybrid")},
        # road-like graph: thousands of levels with a few thousand vertices each
        {"name": "bfs_grid1500", **case("bfs", "grid", 1500 * 1500, direction="hybrid")},
        # the batched engine's full width, as BC-like analyses and the server use it
        {"name": "bfs64_rmat20", **case("batch", "rmat", 1 << 20, sources=64)},
        # the benchmark's SSSP: delta-stepping on float weights in (0, 1]
        {"name": "sssp_rmat22", **case("sssp", "rmat", 1 << 22, delta=0.1)},
        # the reference's schedule (the default) on a directed graph of odd size with integer weights
        {"name": "sssp_directed_u32", **case("sssp", "rmat", 250_001, relabel=True, directed=True, weights="u32",
                                             delta=0.0)},
        # the selector's evaluation grid (2% long-range pairs, integer weights), a quarter of its area
        {"name": "sssp_grid2048", **case("sssp", "grid", 2048 * 2048, long_range=0.02, weights="u32", delta=512.0)},
        # components of a large graph with shuffled ids
        {"name": "cc_rmat3m", **case("cc", "rmat", 3_000_001, relabel=True)},
        # the benchmark's batched betweenness centrality
        {"name": "bc64_rmat20", **case("bc", "rmat", 1 << 20, sources=64, batched=True)},
        # the benchmark's triangle count
        {"name": "tc_rmat20", **case("tc", "rmat", 1 << 20, per_vertex=False)},
        # edge list on the device -> symmetrised, de-duplicated weighted CSR
        {"name": "build_rmat20", **case("build", "rmat", 1 << 20)},
        # a program's own BFS loop on the operators, one advance per level
        {"name": "ops_bfs_300k", **case("ops", "rmat", 300_007, relabel=True, loop="bfs", balancer="workgroup")},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bfs", "batch", "sssp", "cc", "bc", "tc", "build", "ops"])
    graph = rng.choice(["rmat", "rmat", "uniform", "grid"])
    # up to the sizes of the listed cases of the same kind
    top = {"bfs": 1 << 22, "batch": 1 << 20, "sssp": 1 << 22, "cc": 3_000_001, "bc": 1 << 20, "tc": 1 << 20,
           "build": 1 << 20, "ops": 300_007}[kind]
    if graph == "grid":  # long diameters cost a level each: no larger than the listed grids
        top = min(top, {"bfs": 1500 * 1500, "ops": 200 * 200}.get(kind, top))
    n = _log_int(rng, 1 << 10, top)
    long_range = 0.0
    if graph == "grid":
        n = max(32, math.isqrt(n)) ** 2
        long_range = rng.choice([0.0, 0.02])
        if kind in ("batch", "bc", "sssp"):  # their per-level state makes thousands of levels a different workload
            long_range = 0.02
    directed = graph != "grid" and kind != "tc" and rng.random() < 0.4
    c = case(kind, graph, n, rng.randint(4, 16), long_range=long_range, relabel=rng.random() < 0.5, directed=directed,
             weights=rng.choice(["f32", "u32"]))
    if kind == "bfs":
        c["direction"] = rng.choice(["hybrid", "hybrid", "push"])
    elif kind == "batch":
        c["sources"] = rng.randint(1, 64)
    elif kind == "sssp":
        mean = 0.5 if c["weights"] == "f32" else MAX_U32_WEIGHT / 2
        c["delta"] = round(rng.choice([0.0, 0.2 if graph != "grid" else 16.0]) * mean, 3)
    elif kind == "bc":
        c["batched"] = rng.random() < 0.7
        c["sources"] = rng.randint(1, 64) if c["batched"] else rng.randint(1, 3)
    elif kind == "tc":
        c["per_vertex"] = rng.random() < 0.3
    elif kind == "ops":
        c["loop"] = rng.choice(["bfs", "bfs", "sssp"])
        c["balancer"] = rng.choice(["workgroup", "bucketing"])
    return c


# ------------------------------------------------------------------- the graphs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _weights_of(u, v, c, seed):
    """Weights keyed by the pair (of an undirected graph: unordered), so that
    repeated pairs and the two directions of an edge carry the same one."""
    if not c["directed"]:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    x = (u * c["n"] + v) * 0x9E3779B97F4A7C1 + seed * 0x632BE59BD9B4E019 % (1 << 62)
    x = (x ^ (x >> 29)) * 0x3F58476D1CE4E5B9
    x = (x ^ (x >> 32)) * 0x14D049BB133111EB
    x = (x >> 24) & 0xFFFFFF  # 24 random bits
    if c["weights"] == "u32":
        return (1 + x % MAX_U32_WEIGHT).to(torch.int32)
    return (x + 1).to(torch.float32) / float(1 << 24)


def edges(c, seed):
    """The generated edge list: (src, dst, weights), int64 ids on the GPU."""
    g = _generator(seed)
    n = c["n"]
    if c["graph"] == "rmat":
        count = c["degree"] * n
        u = torch.zeros(count, dtype=torch.int64, device="cuda")
        v = torch.zeros_like(u)
        for _ in range(max(1, math.ceil(math.log2(n)))):
            r = torch.rand(count, device="cuda", generator=g)
            u.mul_(2).add_(r >= A + B)
            v.mul_(2).add_(((r >= A) & (r < A + B)) | (r >= A + B + C))
        u %= n
        v %= n
    elif c["graph"] == "uniform":
        count = c["degree"] * n
        u = torch.randint(n, (count,), device="cuda", generator=g)
        v = torch.randint(n, (count,), device="cuda", generator=g)
    else:
        side = math.isqrt(n)
        at = torch.arange(n, device="cuda").view(side, side)
        extra = int(c["long_range"] * 2 * side * (side - 1))
        far = torch.randint(n, (2, extra), device="cuda", generator=g)
        u = torch.cat([at[:, :-1].reshape(-1), at[:-1].reshape(-1), far[0]])
        v = torch.cat([at[:, 1:].reshape(-1), at[1:].reshape(-1), far[1]])
    if c["relabel"]:
        p = torch.randperm(n, device="cuda", generator=g)
        u, v = p[u], p[v]
    return u, v, _weights_of(u, v, c, seed)


class _View:
    """A device array of the library as torch sees it; keeps its owner alive."""

    def __init__(self, ptr, shape, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 2}


def _view(ptr, shape, kind, owner):
    return torch.as_tensor(_View(ptr, shape, kind, owner), device="cuda")


def _result(entry, instance, shape, kind="<i4"):
    p = ctypes.c_void_p()
    call(entry, instance.handle, ctypes.cast(ctypes.pointer(p), getattr(_lib.lib, entry).argtypes[1]))
    return _view(p.value, shape, kind, instance)


def _to_device(t, dtype):
    d = DeviceArray(shape=t.numel(), dtype=dtype)
    call("sg_memcpy", ctypes.c_void_p(d.ptr), ctypes.c_void_p(t.data_ptr()), d.nbytes, 2, None)
    return d


def _edge_arrays(c, seed):
    u, v, w = _build_input(c, seed) if c["kind"] == "build" else edges(c, seed)
    return (_to_device(u.to(torch.int32), np.uint32), _to_device(v.to(torch.int32), np.uint32),
            _to_device(w, np.float32 if c["weights"] == "f32" else np.uint32))


def _build_input(c, seed):
    """An edge list with a known number of distinct pairs (so that the graph
    of every seed has the same size): that many of the generated ones in random
    order, then repeats of some of them, some of those the other way round."""
    u, v, _ = edges(c, seed)
    n, count, g = c["n"], u.numel(), _generator(seed + 5)
    if not c["directed"]:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    key = torch.unique((u * n + v)[u != v])
    distinct = _distinct_pairs(c)
    key = key[torch.randperm(key.numel(), device="cuda", generator=g)[:distinct]]
    assert key.numel() == distinct
    key = torch.cat([key, key[torch.randint(distinct, (count - distinct,), device="cuda", generator=g)]])
    key = key[torch.randperm(count, device="cuda", generator=g)]
    u, v = key // n, key % n
    if not c["directed"]:
        turn = torch.rand(count, device="cuda", generator=g) < 0.5
        u, v = torch.where(turn, v, u), torch.where(turn, u, v)
    return u, v, _weights_of(u, v, c, seed)


def _build(c, arrays):
    return sg.graph.build.fromCOO(c["n"], *arrays, symmetrize=not c["directed"], dedupe=True, drop_self_loops=True)


def _csr(G, c):
    v = G.device_view()
    address = lambda p: ctypes.cast(p, ctypes.c_void_p).value  # noqa: E731
    return {"row_offsets": _view(address(v.row_offsets), (v.n + 1,), "<i4", G),
            "columns": _view(address(v.column_indices), (v.m,), "<i4", G),
            "values": _view(address(v.values), (v.m,), "<f4" if c["weights"] == "f32" else "<i4", G)}


def _sources(G, c, seed):
    """Uniform among the vertices that have an out-edge."""
    ro = _csr(G, c)["row_offsets"]
    some = torch.nonzero(ro[1:] != ro[:-1]).reshape(-1)
    at = torch.randint(some.numel(), (c.get("sources", 1),), device="cuda", generator=_generator(seed + 7))
    return some[at].cpu().numpy().astype(np.uint32)


def prepare(c, seed):
    arrays = _edge_arrays(c, seed)
    if c["kind"] == "build":
        return {"case": c, "arrays": arrays}
    G = _build(c, arrays)
    del arrays
    n = c["n"]
    s = {"case": c, "G": G, "sources": _sources(G, c, seed)}
    s["source"] = int(s["sources"][0])
    kind, alg = c["kind"], sg.algorithms
    if kind == "bfs":
        s["bfs"] = alg.BFS(G)
        s["out"] = _result("sg_bfs_distances_device", s["bfs"], (n,))
    elif kind == "batch":
        s["batch"] = alg.MultiBFS(G, 64)
        s["out"] = _result("sg_msbfs_depths_device", s["batch"], (c["sources"], n))
    elif kind == "sssp":
        s["sssp"] = alg.SSSP(G)
        s["sssp"].set_delta(c["delta"])
        s["out"] = _result("sg_sssp_distances_device", s["sssp"], (n,), "<f4" if c["weights"] == "f32" else "<i4")
    elif kind == "cc":
        s["cc"] = alg.CC(G)
        s["out"] = _result("sg_cc_labels_device", s["cc"], (n,))
    elif kind == "bc" and c["batched"]:
        s["bc"] = alg.BatchedBC(G)
        s["out"] = _result("sg_bc_batch_bc_device", s["bc"], (n,), "<f4")
    elif kind == "bc":
        s["bc"] = alg.BC(G)
    elif kind == "tc":
        s["tc"] = alg.TC(G)
    elif kind == "ops":
        s["in"], s["next"] = sg.frontier.makeFrontier(G), sg.frontier.makeFrontier(G)
        s["out"] = torch.empty(n, dtype=torch.float32 if _float_distances(c) else torch.int32, device="cuda")
        s["mark"] = torch.empty(n, dtype=torch.int32, device="cuda")
    return s


def _float_distances(c):
    return c["weights"] == "f32" and (c["kind"] == "sssp" or c.get("loop") == "sssp")


# --------------------------------------------------------------------- the pass
def run(s):
    c = s["case"]
    return _RUN[c["kind"]](s, c)


def _run_bfs(s, c):
    s["bfs"].init(s["source"])
    mode = sg.algorithms.bfs_direction
    d = s["bfs"].run(mode.hybrid if c["direction"] == "hybrid" else mode.push, ALPHA, BETA)
    return {"depth": s["out"], "levels": d.iterations, "vertices": d.visited_vertices, "edges": d.visited_edges}


def _run_batch(s, c):
    d = s["batch"].run(s["sources"], sg.algorithms.bfs_direction.hybrid, ALPHA_BATCHED, BETA)
    return {"depth": s["out"], "levels": d["iterations"], "edges": d["reached_edges"]}


def _run_sssp(s, c):
    s["sssp"].init(s["source"])
    s["sssp"].run()
    return {"distance": s["out"]}


def _run_cc(s, c):
    s["cc"].run()
    return {"label": s["out"]}


def _run_bc(s, c):
    if c["batched"]:
        s["bc"].run(s["sources"])
        return {"bc": s["out"]}
    s["bc"].init(s["sources"])
    s["bc"].run()
    return {"bc": s["bc"].getBC()}


def _run_tc(s, c):
    s["tc"].run(c["per_vertex"])
    return {"triangles": s["tc"].getNumTriangles(),
            "per_vertex": s["tc"].per_vertex.view(np.int64) if c["per_vertex"] else None}


def _run_build(s, c):
    return _csr(_build(c, s["arrays"]), c)


def _run_ops(s, c):
    """The reference's BFS (or SSSP) loop: advance, (filter,) swap, clear, until the frontier is empty."""
    ops, G, out = sg.operators, s["G"], s["out"]
    balancer = getattr(ops.load_balancer, "workgroup_mapped" if c["balancer"] == "workgroup" else "bucketing")
    n = c["n"]
    now, then = s["in"], s["next"]
    out.fill_(n + 1)
    out[s["source"]] = 0
    now.clear()
    then.clear()
    now.insert(s["source"])
    step = 0
    if c["loop"] == "sssp":
        s["mark"].fill_(-1)
    while not now.empty():
        if c["loop"] == "bfs":
            args = ops.op_args([out.data_ptr()], [n + 1, step])
            ops.advance.frontier(G, now, then, ops.OP_BFS_PUSH, args, ops.direction.push, balancer)
        else:
            args = ops.op_args([out.data_ptr()])
            ops.advance.frontier(G, now, then, ops.OP_SSSP_RELAX, args, ops.direction.push, balancer)
            ops.filter.external(G, then, now, ops.PRED_ITER_MARK, ops.op_args([s["mark"].data_ptr()], [step]))
            sg.frontier.swap(now, then)
        sg.frontier.swap(now, then)
        then.clear()
        step += 1
    return {"distance": out}


_RUN = {"bfs": _run_bfs, "batch": _run_batch, "sssp": _run_sssp, "cc": _run_cc, "bc": _run_bc, "tc": _run_tc,
        "build": _run_build, "ops": _run_ops}


# ------------------------------------------------------------ what a pass needs
def _edge_count(c):
    """Edges of the built graph.  Repeated pairs and self-loops of RMAT take a
    share that was measured on scales 8 to 20 at 4 and 16 pairs per vertex."""
    n, pairs = c["n"], c["degree"] * c["n"]
    if c["graph"] == "grid":
        pairs = 2 * n * (1 + c["long_range"])
    elif c["graph"] == "rmat":
        lost = 0.36 * 0.84 ** (math.log2(n) - 10) * math.sqrt(c["degree"] / 16)
        pairs *= 1 - min(0.6, lost * (0.73 if c["directed"] else 1.0))
    return pairs * (1 if c["directed"] else 2)


def _distinct_pairs(c):
    """Distinct pairs of a construction's input: safely below what is generated."""
    return int(0.85 * _edge_count(c) / (1 if c["directed"] else 2))


def work(c):
    """The graph read once and the results written once; the additions and
    comparisons are one per edge (and source), far below any arithmetic rate."""
    n, m, kind = c["n"], _edge_count(c), c["kind"]
    graph = 4 * (n + 1) + 4 * m
    relaxing = kind == "sssp" or c.get("loop") == "sssp"
    if relaxing:
        return {"bytes": graph + 4 * m + 4 * n, "flops": m}
    if kind == "batch":
        return {"bytes": graph + 4 * n * c["sources"], "flops": 0}
    if kind == "bc":
        return {"bytes": graph + 4 * n, "flops": 2 * m * c["sources"]}
    if kind == "tc":
        return {"bytes": graph + (8 * n if c["per_vertex"] else 8), "flops": 0}
    if kind == "build":
        pairs = 2 * n * (1 + c["long_range"]) if c["graph"] == "grid" else c["degree"] * n
        m = _distinct_pairs(c) * (1 if c["directed"] else 2)
        return {"bytes": 12 * pairs + (2 if c["directed"] else 1) * (4 * (n + 1) + 8 * m), "flops": 0}
    return {"bytes": graph + 4 * n, "flops": 0}


# ------------------------------------------------------------------ its results
def tolerance(c):
    # Depths, labels, counts and the graph are whole numbers; a distance is the
    # least fixed point of rounded sums and so the same bits in any order of
    # relaxation.  Centrality is sums of float32 in some order: 64 sources on
    # RMAT-20 are 2.5e-7 from the 64-bit result.
    return {"rel": 2e-6} if c["kind"] == "bc" else "exact"


def _edges_both_ways(c, seed):
    u, v, w = edges(c, seed)
    w = w.double()
    return (u, v, w) if c["directed"] else (torch.cat([u, v]), torch.cat([v, u]), torch.cat([w, w]))


def exact(c, seed):
    if c["kind"] == "bc":
        return _exact_bc(c, seed)
    if _float_distances(c):
        return _exact_distances(c, seed)
    return None  # whole numbers, or values that are copied


def _seeded_sources(u, v, c, seed):
    has = torch.zeros(c["n"], dtype=torch.bool, device="cuda")
    has[u[u != v]] = True
    some = torch.nonzero(has).reshape(-1)
    return some[torch.randint(some.numel(), (c.get("sources", 1),), device="cuda", generator=_generator(seed + 7))]


def _exact_distances(c, seed):
    """Bellman-Ford over every edge until nothing changes."""
    u, v, w = _edges_both_ways(c, seed)
    n = c["n"]
    d = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    d[_seeded_sources(u, v, c, seed)[0]] = 0
    while True:
        new = d.scatter_reduce(0, v, d[u] + w, "amin")
        if torch.equal(new, d):
            break
        d = new
    return {"distance": torch.where(torch.isinf(d), torch.full_like(d, n + 1), d)}


def _exact_bc(c, seed):
    """Brandes, a source at a time: path counts forward, dependencies backward."""
    u, v, _ = _edges_both_ways(c, seed)
    n = c["n"]
    sources = _seeded_sources(u, v, c, seed).tolist()
    key = torch.unique(u * n + v)
    u, v = key // n, key % n
    del key
    bc = torch.zeros(n, dtype=torch.float64, device="cuda")
    for s in sources:
        depth = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        depth[s] = 0
        sigma = torch.zeros(n, dtype=torch.float64, device="cuda")
        sigma[s] = 1
        levels, at = [], 0
        while True:
            e = torch.nonzero((depth[u] == at) & (depth[v] == -1)).reshape(-1)
            if not e.numel():
                break
            a, b = u[e], v[e]
            depth[b] = at + 1
            sigma.index_add_(0, b, sigma[a])
            levels.append((a, b))
            at += 1
        delta = torch.zeros_like(sigma)
        for a, b in reversed(levels):
            delta.index_add_(0, a, sigma[a] / sigma[b] * (1 + delta[b]))
        delta[s] = 0
        bc += delta
    return {"bc": bc}

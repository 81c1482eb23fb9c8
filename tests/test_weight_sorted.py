"""The weight-sorted adjacency of delta-stepping SSSP, built on the device
(sg_graph_weight_sorted): every row holds the same (column, weight) pairs as
the CSR, in non-decreasing weight order with equal weights in column order,
and the symmetry flag is right."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def host_sorted(g):
    ro, col, val = g.row_offsets, g.column_indices, g.values
    bits = val.view(np.uint32) if val.dtype == np.float32 else val
    rows = np.repeat(np.arange(g.n, dtype=np.uint64), np.diff(ro.astype(np.int64)))
    order = np.lexsort((col, bits, rows))  # by row, then weight, then column
    return col[order], val[order]


@pytest.mark.parametrize("kind", ["rmat_f32", "rmat_u32", "grid_u32", "directed", "asym_weights"])
def test_weight_sorted_rows(sg, rmat, kind):
    props = None
    if kind == "rmat_f32":
        g = rmat(16, perm_seed=3)
    elif kind == "rmat_u32":
        g = rmat(14, value_type=sg.WEIGHT_U32)
    elif kind == "grid_u32":
        g = sg.io.grid(200, 0.02, value_type=sg.WEIGHT_U32)
    else:
        rng = np.random.default_rng(7)
        n, k = 3000, 40000
        s, d = rng.integers(0, n, k), rng.integers(0, n, k)
        w = rng.integers(1, 9, k).astype(np.uint32)
        if kind == "directed":
            g = sg.io.fromCOO(n, s, d, w, dedupe=True, drop_self_loops=True)
            props = sg.Properties(directed=True, weighted=True)
        else:  # symmetric pattern, weights differ by direction
            g = sg.io.fromCOO(n, np.concatenate([s, d]), np.concatenate([d, s]),
                              np.concatenate([w, w + 1]), dedupe=True, drop_self_loops=True)
    G = sg.graph.build.fromCSR(g, props)
    col, val, sym = G.weight_sorted()
    want_col, want_val = host_sorted(g)
    assert np.array_equal(col, want_col)
    assert np.array_equal(val.view(np.uint32), want_val.view(np.uint32))
    assert sym == kind.startswith(("rmat", "grid"))


@pytest.mark.parametrize("n", [2, 33, 500])
@pytest.mark.parametrize("broken", ["none", "missing", "weight", "both_missing", "self_loop"])
def test_weight_symmetry_flag(sg, n, broken):
    """The flag looks one direction of every pair up and counts the other: a
    reverse missing towards either end, a weight that differs, and self-loops
    (their own reverse)."""
    rng = np.random.default_rng(n)
    a = np.arange(n - 1)
    s, d = np.concatenate([a, np.zeros(n - 1, int)]), np.concatenate([a + 1, a + 1])  # a path and a star on 0
    pairs = sorted({(min(x, y), max(x, y)) for x, y in zip(s, d)})
    w = rng.integers(1, 50, len(pairs))
    edges = {(x, y): k for (x, y), k in zip(pairs, w)} | {(y, x): k for (x, y), k in zip(pairs, w)}
    if broken == "missing":  # towards the larger end (vertex 0) of one pair
        del edges[(pairs[-1][1], pairs[-1][0])]
    elif broken == "both_missing" and len(pairs) > 1:  # one towards each end, of different pairs
        del edges[pairs[0]]
        del edges[(pairs[-1][1], pairs[-1][0])]
    elif broken == "weight":
        edges[pairs[0]] += 1
    elif broken == "self_loop":
        edges[(n // 2, n // 2)] = 7
    e = sorted(edges)
    ro = np.searchsorted([x for x, _ in e], np.arange(n + 1)).astype(np.uint32)
    g = sg.CSR(ro, np.array([y for _, y in e], np.uint32), np.array([edges[x] for x in e], np.uint32))
    G = sg.graph.build.fromCSR(g)
    col, val, sym = G.weight_sorted()
    want_col, want_val = host_sorted(g)
    assert np.array_equal(col, want_col) and np.array_equal(val, want_val)
    bits = {(x, y): k for (x, y), k in edges.items()}
    assert sym == all(bits.get((y, x)) == k for (x, y), k in bits.items())


@pytest.mark.parametrize("gap", [0, 31, 200, 12_000_000])
def test_weight_sorted_rows_across_empty_rows(sg, gap):
    """Long runs of vertices without edges, inside and between the words of 32
    edges that a warp takes: the same rows, and no time spent on the run (a
    warp that passes it 32 rows at a time takes 0.15 s for the longest one)."""
    k, half = 80, 40
    n = k + 12_000_000
    ids = np.concatenate([np.arange(half), half + gap + np.arange(half)])
    deg = np.zeros(n, np.int64)
    deg[ids] = k - 1
    ro = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    i, j = np.nonzero(~np.eye(k, dtype=bool))
    g = sg.CSR(ro, ids[j].astype(np.uint32), (1 + (i * j) % 7).astype(np.uint32))
    want_col, want_val = host_sorted(g)
    seconds = []
    for _ in range(3):
        G = sg.graph.build.fromCSR(g)
        t = time.perf_counter()
        col, val, sym = G.weight_sorted()
        seconds.append(time.perf_counter() - t)
        assert np.array_equal(col, want_col) and np.array_equal(val, want_val) and sym
    assert min(seconds) < 0.05

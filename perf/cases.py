"""What this library's users have it do, as a list of cases that can be timed and checked.

Each case is one call (or one batch of queries) through the public Python entry points:
single-source shortest paths with the three methods, dense min-plus products, all-pairs
shortest paths, sparse min-plus products and the query server.  Graph families, weight laws
and sizes are those of the benchmark and the tests: symmetrised RMAT (edge factor 16, weights
U{1..255}), road-like grids with 2 % random long-range pairs (lognormal weights), directed
Erdos-Renyi graphs (weights U{1..100}), 30 % dense matrices.  Inputs are made on the GPU from
the seed alone.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs and handles a program holds before the call
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the floating outputs in 64 bits, by plain torch
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rips2026-amd_b200"))
import b200sssp  # noqa: E402
from b200sssp.serving import Server  # noqa: E402

MISSING = (2**31 - 1) // 2   # "no entry" of an int32 min-plus matrix


def listed():
    return [
        # The smallest solve of the benchmark: a 4096-vertex random graph, where launch and phase
        # latency is all there is.
        {"name": "bf_er4096_u32", "kind": "sssp", "graph": "er", "n": 4096, "degree": 8, "method": "bf",
         "weight": "u32", "pred": False},
        # Bellman-Ford with predecessors on a mid-size skewed graph, float weights.
        {"name": "bf_rmat17_f32_pred", "kind": "sssp", "graph": "rmat", "scale": 17, "method": "bf", "weight": "f32",
         "pred": True},
        # An ordinary road-like query that wants the path back: many small frontiers.
        {"name": "delta_grid_u32_pred", "kind": "sssp", "graph": "grid", "rows": 411, "cols": 300, "method": "delta",
         "weight": "u32", "pred": True},
        # The headline: delta-stepping on RMAT scale 24 (16.8 M vertices, 0.5 G arcs).
        {"name": "delta_rmat24_u32", "kind": "sssp", "graph": "rmat", "scale": 24, "method": "delta", "weight": "u32",
         "pred": False},
        # The other large graph of the benchmark, with its float weights: a 16.8 M-vertex grid.
        {"name": "delta_grid4096_f32", "kind": "sssp", "graph": "grid", "rows": 4096, "cols": 4096, "method": "delta",
         "weight": "f32", "pred": False},
        # The asynchronous worklist on a mid-size skewed graph.
        {"name": "adds_rmat18_u32", "kind": "sssp", "graph": "rmat", "scale": 18, "method": "adds", "weight": "u32",
         "pred": False},
        # The dense product of the benchmark.
        {"name": "gemm_f32_8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "dtype": "f32"},
        # A ragged product: no size a multiple of a tile, rows that do not start on 16 bytes.
        {"name": "gemm_i32_ragged", "kind": "gemm", "m": 1111, "n": 1503, "k": 777, "dtype": "i32"},
        # All pairs of a sparse graph of a thousand vertices.
        {"name": "apsp_f32_1000", "kind": "apsp", "n": 1000, "degree": 8, "dtype": "f32"},
        # The sparse product of the benchmark: 2^20 rows of about 8 entries, about 64 candidates a row.
        {"name": "spgemm_er20_i32", "kind": "spgemm", "graph": "er", "n": 1 << 20, "degree": 8, "dtype": "i32"},
        # A sparse product of a skewed matrix: rows from a few to many thousands of candidates.
        {"name": "spgemm_rmat14_f32", "kind": "spgemm", "graph": "rmat", "scale": 14, "edge_factor": 8, "dtype": "f32"},
        # The server: a burst of queries over resident graphs of uneven size.
        {"name": "serve_9graphs_256q", "kind": "serve", "queries": 256, "max_grid": 1024, "max_scale": 18},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sssp", "sssp", "sssp", "gemm", "gemm", "apsp", "spgemm", "serve"])
    if kind == "sssp":
        method = rng.choice(["delta", "delta", "bf", "adds"])
        case = {"kind": "sssp", "graph": rng.choice(["er", "rmat", "grid"]), "method": method,
                "weight": rng.choice(["u32", "f32"]), "pred": rng.random() < 0.3}
        if case["graph"] == "er":
            case.update(n=_log_int(rng, 1000, 1 << 20), degree=rng.randint(4, 16))
        elif case["graph"] == "rmat":
            case.update(scale=rng.randint(10, 22 if method == "delta" else 19))
        else:
            top = {"delta": 2048, "bf": 256, "adds": 1024}[method]
            case.update(rows=_log_int(rng, 40, top), cols=_log_int(rng, 40, top))
        return case
    if kind == "gemm":
        return {"kind": "gemm", "m": _log_int(rng, 60, 4500), "n": _log_int(rng, 60, 4500), "k": _log_int(rng, 60, 4500),
                "dtype": rng.choice(["f32", "i32"])}
    if kind == "apsp":
        return {"kind": "apsp", "n": _log_int(rng, 100, 3000), "degree": rng.randint(3, 30),
                "dtype": rng.choice(["f32", "i32"])}
    if kind == "spgemm":
        if rng.random() < 0.5:
            return {"kind": "spgemm", "graph": "er", "n": _log_int(rng, 3000, 1 << 20), "degree": rng.randint(3, 12),
                    "dtype": rng.choice(["f32", "i32"])}
        return {"kind": "spgemm", "graph": "rmat", "scale": rng.randint(9, 15), "edge_factor": rng.randint(4, 8),
                "dtype": rng.choice(["f32", "i32"])}
    return {"kind": "serve", "queries": _log_int(rng, 16, 256), "max_grid": rng.choice([256, 512, 1024]),
            "max_scale": rng.randint(13, 18)}


# ---------------------------------------------------------------------------
# inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _csr(n, u, v, w):
    """Outgoing CSR (int64 row pointers, int32 columns, weights) of arcs with distinct (u, v)."""
    key, order = torch.sort(u * n + v)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(u, minlength=n), 0)
    return rowptr, (key % n).to(torch.int32), w[order]


def _er(n, degree, gen):
    m = n * degree
    key = torch.randint(0, n * n, (m,), device="cuda", generator=gen)
    key = torch.unique(key)
    u, v = key // n, key % n
    keep = u != v
    u, v = u[keep], v[keep]
    return n, u, v, torch.randint(1, 101, (u.numel(),), device="cuda", generator=gen, dtype=torch.int32), 101.0


def _rmat(scale, edge_factor, gen):
    n = 1 << scale
    m = n * edge_factor
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, device="cuda", generator=gen)
        u.mul_(2).add_(r >= 0.76)
        v.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    # spread the hubs over the id range
    scramble = torch.randint(0, n, (2,), generator=gen, device="cuda")
    mul, add = (scramble[0] | 1), scramble[1]
    u.mul_(mul).add_(add).bitwise_and_(n - 1)
    v.mul_(mul).add_(add).bitwise_and_(n - 1)
    lo, hi = torch.minimum(u, v), torch.maximum(u, v)
    del u, v
    key = lo.mul_(n).add_(hi)[lo.div(n, rounding_mode="floor") != hi]
    del lo, hi
    key = torch.unique(key)
    w = torch.randint(1, 256, (key.numel(),), device="cuda", generator=gen, dtype=torch.int32)
    a, b = key // n, key % n
    return n, torch.cat([a, b]), torch.cat([b, a]), torch.cat([w, w]), 256.0


def _grid(rows, cols, gen):
    n = rows * cols
    at = torch.arange(n, device="cuda").view(rows, cols)
    a = [at[:, :-1].reshape(-1), at[:-1].reshape(-1)]
    b = [at[:, 1:].reshape(-1), at[1:].reshape(-1)]
    pairs = int(round(0.02 * 2 * (a[0].numel() + a[1].numel())))
    far = torch.randint(0, n, (2, pairs), device="cuda", generator=gen)
    a = torch.cat(a + [far[0]])
    b = torch.cat(b + [far[1]])
    key = torch.unique(torch.cat([a * n + b, b * n + a]))
    u, v = key // n, key % n
    keep = u != v
    u, v = u[keep], v[keep]
    w = torch.randn(u.numel(), device="cuda", generator=gen).add_(5.0).exp_().ceil_().clamp_(1.0, 1e6)
    return n, u, v, w.to(torch.int32), 30000.0


def _arcs(case, gen):
    if case["graph"] == "er":
        return _er(case["n"], case["degree"], gen)
    if case["graph"] == "rmat":
        return _rmat(case["scale"], case.get("edge_factor", 16), gen)
    return _grid(case["rows"], case["cols"], gen)


def _graph_csr(case, seed):
    """CSR with the case's weights (uint32, or the same law scaled towards [0, 1)) and a source that has arcs."""
    gen = _generator(seed)
    n, u, v, w, scale = _arcs(case, gen)
    if case.get("weight", "u32") == "f32":
        w = w.to(torch.float32).div_(scale)
    rowptr, colind, w = _csr(n, u, v, w)
    source = int(colind[int(torch.randint(0, colind.numel(), (1,), device="cuda", generator=gen))])
    return rowptr, colind, w, source


def _dense(rows, cols, dtype, gen):
    """30 % of the entries present."""
    present = torch.rand(rows, cols, device="cuda", generator=gen) < 0.3
    if dtype == "f32":
        return torch.where(present, torch.rand(rows, cols, device="cuda", generator=gen), math.inf)
    return torch.where(present, torch.randint(1, 1001, (rows, cols), device="cuda", generator=gen, dtype=torch.int32),
                       MISSING)


def _adjacency(case, seed):
    """Dense distance matrix of a random directed graph: zero diagonal, missing arcs absent."""
    gen = _generator(seed)
    n = case["n"]
    present = torch.rand(n, n, device="cuda", generator=gen) < case["degree"] / n
    if case["dtype"] == "f32":
        d = torch.where(present, torch.rand(n, n, device="cuda", generator=gen), math.inf)
    else:
        d = torch.where(present, torch.randint(1, 1001, (n, n), device="cuda", generator=gen, dtype=torch.int32), MISSING)
    d.fill_diagonal_(0)
    return d


def _sparse(case, seed):
    """(rowptr, colind, values, columns) of a square matrix.  The seed renumbers the vertices of one
    random graph and draws the values, so that the product has as many entries for every seed."""
    n, u, v, w, scale = _arcs(case, _generator(1))
    gen = _generator(seed)
    order = torch.randperm(n, device="cuda", generator=gen)
    w = w[torch.randperm(w.numel(), device="cuda", generator=gen)]
    if case["dtype"] == "f32":
        w = w.to(torch.float32).div_(scale)
    return (*_csr(n, order[u], order[v], w), n)


def _served_graphs(case):
    """Grids and RMAT graphs from small to the case's largest."""
    graphs = [{"graph": "grid", "rows": s, "cols": s} for s in (64, 128, 256, 512, 1024) if s <= case["max_grid"]]
    return graphs + [{"graph": "rmat", "scale": s} for s in (12, 14, 16, 18) if s <= case["max_scale"]]


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "sssp":
        rowptr, colind, w, source = _graph_csr(case, seed)
        g = b200sssp.Graph.from_arrays(rowptr, colind, w, weight=case["weight"])
        return {"kind": kind, "graph": g, "source": source, "method": case["method"], "pred": case["pred"]}
    if kind == "gemm":
        gen = _generator(seed)
        return {"kind": kind, "a": _dense(case["m"], case["k"], case["dtype"], gen),
                "b": _dense(case["k"], case["n"], case["dtype"], gen)}
    if kind == "apsp":
        d = _adjacency(case, seed)
        return {"kind": kind, "adjacency": d, "d": torch.empty_like(d)}
    if kind == "spgemm":
        return {"kind": kind, "a": _sparse(case, seed)}
    server = Server(hbm_budget=4 << 30)
    graphs, ids, results, sources = [], [], [], []
    gen = _generator(seed)
    spec = _served_graphs(case)
    # as many queries for each graph, in random order
    pick = (torch.randperm(case["queries"], device="cuda", generator=gen) % len(spec)).tolist()
    for k, c in enumerate(spec):
        rowptr, colind, w, _ = _graph_csr(c, seed * 16 + k)
        g = b200sssp.Graph.from_arrays(rowptr, colind, w, weight="u32")
        graphs.append(g)
        ids.append(server.add_graph(g))
        count = pick.count(k)
        results.append(torch.empty((count, g.n), dtype=torch.int32).pin_memory())
        at = torch.randint(0, colind.numel(), (count,), device="cuda", generator=gen)
        sources.append(colind[at].tolist())   # vertices with arcs
    # queries in arrival order: (graph id, source, result row)
    seen = [0] * len(spec)
    queries = []
    for k in pick:
        queries.append((ids[k], sources[k][seen[k]], results[k][seen[k]]))
        seen[k] += 1
    return {"kind": kind, "server": server, "graphs": graphs, "queries": queries, "results": results}


def run(state):
    kind = state["kind"]
    if kind == "sssp":
        dist, pred, _ = state["graph"].sssp(state["source"], method=state["method"], pred=state["pred"])
        return [dist, pred] if state["pred"] else [dist]
    if kind == "gemm":
        return b200sssp.minplus_gemm(state["a"], state["b"])
    if kind == "apsp":
        state["d"].copy_(state["adjacency"])   # the call works in place
        b200sssp.apsp(state["d"])
        return state["d"]
    if kind == "spgemm":
        return list(b200sssp.minplus_spgemm(state["a"], state["a"]))
    server = state["server"]
    for graph_id, source, out in state["queries"]:
        server.submit(graph_id, source, out)
    server.progress(wait_all=True)
    for done in server.poll():
        if done["status"] != 0:
            raise RuntimeError(f"query {done['ticket']} failed with status {done['status']}")
    return state["results"]


# ---------------------------------------------------------------------------
def _size(case):
    """(vertices, arcs) of a case's graph, about."""
    if case["graph"] == "er":
        return case["n"], case["n"] * case["degree"]
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        return n, int(2 * 0.95 * n * case.get("edge_factor", 16))
    n = case["rows"] * case["cols"]
    return n, int(4.16 * n)


def work(case):
    kind = case["kind"]
    if kind == "sssp":
        # every arc (column, weight) and row pointer read once, the distances (and predecessors) written once
        n, m = _size(case)
        return {"bytes": 8 * m + 8 * n + (8 if case["pred"] else 4) * n, "flops": m}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    if kind == "apsp":
        return {"bytes": 8 * case["n"] ** 2, "flops": 2 * case["n"] ** 3}
    if kind == "spgemm":
        n, m = _size(case)
        if case["graph"] == "er":
            candidates = m * case["degree"]
        else:
            candidates = m * m / n * 2.2 ** (case["scale"] / 4)   # squared degrees of a skewed graph, about
        return {"bytes": 16 * n + 8 * m + 8 * min(candidates, n * n), "flops": candidates}
    total = 0
    spec = _served_graphs(case)
    for c in spec:
        n, m = _size(c)
        total += case["queries"] / len(spec) * (8 * m + 12 * n)
    return {"bytes": int(total), "flops": int(total / 8)}


# ---------------------------------------------------------------------------
# 64-bit results by plain torch
def _exact_sssp(case, seed):
    rowptr, colind, w, source = _graph_csr(case, seed)
    n = rowptr.numel() - 1
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), rowptr[1:] - rowptr[:-1])
    v, w = colind.long(), w.double()
    d = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    d[source] = 0.0
    while True:
        nxt = d.scatter_reduce(0, v, d[u] + w, "amin")
        if torch.equal(nxt, d):
            return d
        d = nxt


def _exact_gemm(case, seed):
    s = prepare(case, seed)
    a, b = s["a"].double(), s["b"].double()
    c = torch.full((case["m"], case["n"]), math.inf, dtype=torch.float64, device="cuda")
    t = torch.empty_like(c)
    for k in range(case["k"]):
        torch.add(a[:, k: k + 1], b[k: k + 1], out=t)
        torch.minimum(c, t, out=c)
    return c


def _exact_apsp(case, seed):
    d = _adjacency(case, seed).double()
    for k in range(case["n"]):
        d = torch.minimum(d, d[:, k: k + 1] + d[k: k + 1])
    return d


def _exact_spgemm(case, seed):
    rowptr, colind, val, n = _sparse(case, seed)
    degree = rowptr[1:] - rowptr[:-1]
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), degree)
    col = colind.long()
    length = degree[col]   # candidates of each entry of A
    entry = torch.repeat_interleave(torch.arange(col.numel(), device="cuda"), length)
    first = torch.cumsum(length, 0) - length
    at = rowptr[col][entry] + torch.arange(entry.numel(), device="cuda") - first[entry]
    key = row[entry] * n + col[at]
    cand = val.double()[entry] + val.double()[at]
    del at, entry
    key, place = torch.unique(key, return_inverse=True)   # in row order, columns ascending
    out = torch.full((key.numel(),), math.inf, dtype=torch.float64, device="cuda")
    return out.scatter_reduce(0, place, cand, "amin")


def exact(case, seed):
    kind = case["kind"]
    if kind == "sssp" and case["weight"] == "f32":
        if case["graph"] == "grid" and case["rows"] * case["cols"] > 1 << 20:
            return None   # thousands of rounds over millions of arcs
        d = _exact_sssp(case, seed)
        return [d, None] if case["pred"] else [d]
    if kind == "gemm" and case["dtype"] == "f32":
        return _exact_gemm(case, seed)
    if kind == "apsp" and case["dtype"] == "f32":
        return _exact_apsp(case, seed)
    if kind == "spgemm" and case["dtype"] == "f32":
        return [None, None, _exact_spgemm(case, seed)]
    return None

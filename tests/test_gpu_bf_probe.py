"""GPU Bellman-Ford predecessors where a hop limit cuts the solve, with and without the
negative-cycle probe, word for word against rounds done one after the other on the CPU.

A vertex's predecessor is the smallest one of the round that last lowered its distance;
later rounds that reach it at the same distance lower the predecessor too, except in the
output of a solve that ended with the probe.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
INF = np.uint64(0xFFFFFFFF)


def _rounds(n, u, v, w, source, limit, probe):
    """(distances, predecessors, rounds) of frontier rounds over packed (distance, predecessor) words."""
    full = np.full(n, ~np.uint64(0))
    full[source] = INF
    last = full.copy()   # as of each vertex's last improvement
    changed = np.zeros(n, bool)
    changed[source] = True
    for k in range(1, limit + 1):
        on = changed[u]
        dist = full >> np.uint64(32)
        word = ((dist[u[on]] + w[on]) << np.uint64(32)) | u[on].astype(np.uint64)
        np.minimum.at(full, v[on], word)
        changed = (full >> np.uint64(32)) < dist
        last[changed] = full[changed]
        if not changed.any():
            break
    out = last if probe and changed.any() else full
    d = (out >> np.uint64(32)).astype(np.uint32)
    p = (out & INF).astype(np.int64)
    p[(d == 0xFFFFFFFF) | (np.arange(n) == source)] = -1
    return d, p.astype(np.int32), k


def _graph(kind):
    rng = np.random.default_rng(6)
    if kind == "ties":      # few distinct weights: most vertices are reached equally from several sides
        n = 3000
        key = np.unique(rng.integers(0, n * n, 20000))
        u, v = key // n, key % n
        w = rng.integers(1, 4, u.size)
    else:                   # rows on both sides of the chunked-row limit (256 edges)
        n = 1500
        u = np.concatenate([np.repeat([3, 700, 1100], [257, 600, 255]), rng.integers(0, n, 9000)])
        v = np.concatenate([np.arange(257) + 20, np.arange(600) + 100, np.arange(255) + 900, rng.integers(0, n, 9000)])
        key = np.unique(u * n + v)
        u, v = key // n, key % n
        w = rng.integers(1, 3, u.size)
    keep = u != v
    return n, u[keep], v[keep], w[keep].astype(np.uint64)


@pytest.mark.parametrize("kind", ["ties", "rows"])
@pytest.mark.parametrize("weight", ["u32", "f32"])
@pytest.mark.parametrize("probe", [0, 1])
def test_predecessors_of_cut_rounds(b2, cuda, kind, weight, probe):
    n, u, v, w = _graph(kind)
    rp = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))]).astype(np.int64)
    g = b2.Graph.from_arrays(rp, v.astype(np.int32), w.astype(np.uint32 if weight == "u32" else np.float32),
                             weight=weight)
    for source in (3, 11):
        for limit in (1, 2, 3, 4, 5, 7, 40):
            d, p, used = _rounds(n, u, v, w, source, limit, probe)
            gd, gp, st = g.sssp(source, method="bf", pred=True, max_iters=limit, detect_negative_cycle=probe)
            assert np.array_equal(b2.dist_to_numpy(gd, weight), np.where(d == 0xFFFFFFFF, np.inf, d.astype(np.float64)))
            assert np.array_equal(gp.cpu().numpy(), p)
            assert st["iterations_used"] == used
    g.close()

"""GPU Bellman-Ford rounds with two label arrays: word for word against the oracle's
Jacobi rounds where a hop limit cuts them, and against Dijkstra where it does not.

uint32 and float32 distances are exact: every label is the minimum of the same
left-to-right sums.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, arcs):
    """Outgoing CSR of (u, v, w) triples."""
    arcs = sorted(arcs)
    rp = np.zeros(n + 1, np.int64)
    for u, _, _ in arcs:
        rp[u + 1] += 1
    return np.cumsum(rp), np.array([a[1] for a in arcs], np.int32), np.array([a[2] for a in arcs])


def _incoming(n, arcs):
    rp, ci, w = _csr(n, [(v, u, x) for u, v, x in arcs])
    return rp, ci, w.astype(np.float32)


def _graphs():
    rng = np.random.default_rng(8)
    # rows on both sides of the chunked-row limit (256 edges) and of one chunk more, the
    # source's own row among them, with equal distances over several predecessors
    for deg in (255, 256, 257, 511, 512, 513, 3000):
        n = deg + 400
        arcs = [(0, i + 1, 1 + i % 3) for i in range(deg)]
        arcs += [(1 + int(u), deg + 1 + int(v), 1 + int(x)) for u, v, x in
                 zip(rng.integers(0, deg, 900), rng.integers(0, 300, 900), rng.integers(0, 3, 900))]
        hub = deg + 1 + 7
        arcs += [(5, hub, 1)] + [(hub, 1 + i, 1) for i in range(deg)] + [(hub, deg + 310 + i % 80, 2) for i in range(300)]
        yield f"hub{deg}", n, list({(u, v): (u, v, x) for u, v, x in arcs if u != v}.values())
    # long chains with shortcuts: labels fall in many rounds; equal ties everywhere
    arcs = [(i, i + 1, 2) for i in range(600)] + [(i, min(i + int(k), 600), 2 * int(k)) for i, k in
                                                  enumerate(rng.integers(2, 40, 560))]
    yield "chain", 601, list({(u, v): (u, v, x) for u, v, x in arcs if u != v}.values())


GRAPHS = {name: (n, arcs) for name, n, arcs in _graphs()}


@pytest.mark.parametrize("name", GRAPHS)
@pytest.mark.parametrize("weight", ["u32", "f32"])
def test_fixpoint_and_predecessors(b2, orc, cuda, name, weight):
    n, arcs = GRAPHS[name]
    rp, ci, w = _csr(n, arcs)
    w = w.astype(np.uint32 if weight == "u32" else np.float32)
    g = b2.Graph.from_arrays(rp, ci, w, weight=weight)
    for s in (0, 5):
        ref = orc.dijkstra(rp, ci, w, s)
        d, _, st = g.sssp(s, method="bf")
        assert np.array_equal(d.cpu().numpy().view(np.uint32), np.ascontiguousarray(ref).view(np.uint32))
        d, p, sp = g.sssp(s, method="bf", pred=True, collect_reach=1)
        assert np.array_equal(d.cpu().numpy().view(np.uint32), np.ascontiguousarray(ref).view(np.uint32))
        assert st["iterations_used"] == sp["iterations_used"] and st["converged"] and sp["converged"]
        reached = np.isfinite(ref) if weight == "f32" else ref != 0xFFFFFFFF
        assert sp["reached"] == int(reached.sum())
        # among the predecessors at equal distance the smallest id
        best = np.full(n, n, np.int64)
        u = np.repeat(np.arange(n), np.diff(rp))
        r64 = ref.astype(np.float64) if weight == "f32" else np.where(reached, ref.astype(np.float64), np.inf)
        tight = reached[u] & (r64[u] + w.astype(np.float64) == r64[ci])
        np.minimum.at(best, ci[tight], u[tight])
        best[best == n] = -1
        best[s] = -1
        assert np.array_equal(p.cpu().numpy(), best)
    g.close()


# odd and even numbers of rounds end in either array
@pytest.mark.parametrize("name", ["hub256", "hub3000", "chain"])
@pytest.mark.parametrize("rounds", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("probe", [False, True])
def test_hop_limited_rounds(b2, orc, cuda, name, rounds, probe):
    n, arcs = GRAPHS[name]
    rp, ci, w = _csr(n, arcs)
    irp, ici, iw = _incoming(n, arcs)
    g = b2.Graph.from_arrays(rp, ci, w.astype(np.float32), weight="f32")
    od, oused, oconv, oneg, _ = orc.bf_jacobi(irp, ici, iw, 0, rounds, detect_negative=probe)
    for pred in (False, True):
        d, p, st = g.sssp(0, method="bf", pred=pred, max_iters=rounds, detect_negative_cycle=int(probe),
                          collect_reach=1)
        got = d.cpu().numpy()
        assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(od, np.float32).view(np.uint32))
        assert st["iterations_used"] == oused and bool(st["converged"]) == bool(oconv)
        assert st["reached"] == int(np.isfinite(od).sum())
    g.close()

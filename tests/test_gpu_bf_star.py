"""GPU Bellman-Ford from a source whose row alone is most of the graph: its chunks are listed
by all threads, so the first phase ends as soon as with a delta-stepping solve of the same row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows one chunk short of, at and past the number of threads that list chunks, and the largest
@pytest.mark.parametrize("leaves", [256, 257, 256 * 75776, 256 * 75777 + 5, 1 << 25])
def test_star_from_its_centre(b2, cuda, leaves):
    torch = cuda
    n = leaves + 1
    rp = torch.full((n + 1,), leaves, dtype=torch.int64, device="cuda")
    rp[0] = 0
    ci = torch.arange(1, n, dtype=torch.int32, device="cuda")
    w = torch.arange(leaves, dtype=torch.int32, device="cuda").remainder_(251).add_(1)
    g = b2.Graph.from_arrays(rp, ci, w, weight="u32")
    best = {}
    for method in ("bf", "delta"):
        d, p, _ = g.sssp(0, method=method, pred=True)
        assert int(d[0]) == 0 and torch.equal(d[1:], w)
        assert int(p[0]) == -1 and int(p[1:].abs().max()) == 0
        best[method] = min(g.sssp(0, method=method)[2]["kernel_ms"] for _ in range(7))
    if leaves == 1 << 25:
        # measured 0.92 (1.25 with one thread listing the chunks)
        assert best["bf"] < 1.1 * best["delta"], best
    g.close()

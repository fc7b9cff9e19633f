"""GPU server: a burst of queries on a graph that is big by its edges alone goes to single blocks,
a few queries to a cluster, and both give Dijkstra's distances word for word."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernels(torch, f):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    names = {e.name for e in p.events()}
    if not any("k_" in n for n in names):
        return None   # no profiler here
    return {k for k in ("k_serve_cluster", "k_serve(") if any(k in n for n in names)}


# 2^15 vertices of uneven degree (blocks from 35 waiting queries on); one lane takes one kind at a time
@pytest.mark.parametrize("lanes", [16, 1])
@pytest.mark.parametrize("pred", [False, True])
def test_bursts_go_to_blocks(b2, orc, cuda, lanes, pred):
    torch = cuda
    from b200sssp.serving import Server
    h = b2.gen_rmat(15, 100, seed=1)
    assert h.m >= 1 << 22 and np.diff(h.rowptr).max() >= 64 * h.m / h.n
    g = b2.Graph.from_host(h, "u32")
    srv = Server(hbm_budget=2 << 30, lanes=lanes)
    gid = srv.add_graph(g)
    assert srv.graph_config(gid)["cluster_team"]
    sources = [int(s) for s in h.colind[:: h.m // 7][:7]]
    refs = [orc.dijkstra(h.rowptr, h.colind, h.weights, s) for s in sources]

    def burst(queries):
        outs = [torch.empty(g.n, dtype=torch.int32).pin_memory() for _ in range(queries)]
        preds = [torch.empty(g.n, dtype=torch.int32).pin_memory() if pred else None for _ in range(queries)]

        def run():
            for k in range(queries):
                srv.submit(gid, sources[k % 7], outs[k], preds[k])
            srv.progress(wait_all=True)
        used = _kernels(torch, run)
        done = srv.poll()
        assert len(done) == queries and all(c["status"] == 0 for c in done)
        for k in range(queries):
            assert np.array_equal(outs[k].numpy().view(np.uint32), refs[k % 7])
            if pred and k < 7:
                assert orc.validate_spt(h.rowptr, h.colind, h.weights, sources[k], outs[k].numpy().view(np.uint32),
                                        preds[k].numpy()) == 0
        return used

    burst(2)   # (the profiler and the lanes' graphs are set up)
    assert burst(34) in (None, {"k_serve_cluster"})
    assert burst(60) in (None, {"k_serve("})
    srv.close()
    g.close()

"""GPU server: the team of a graph follows its vertices and its edges, and both
teams give Dijkstra's distances word for word."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 2^22 edges on either side of the default rule, below 2^19 vertices, with rows on
# both sides of the length that a whole team relaxes together; big_vertices < 0 and
# a vertex count of one's own leave the edges out of it
@pytest.mark.parametrize("arcs,big_vertices,cluster", [((1 << 22) - 1, 0, False), (1 << 22, 0, True),
                                                       (1 << 22, -1, False), (1 << 22, 1 << 20, False)])
def test_team_follows_edges(b2, orc, cuda, arcs, big_vertices, cluster):
    from b200sssp.serving import Server
    n = 30000
    rng = np.random.default_rng(arcs & 7)
    u = rng.integers(0, n, arcs)
    u[:3000] = 17
    v = rng.integers(0, n, arcs)
    order = np.argsort(u, kind="stable")
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(u, minlength=n))
    ci = v[order].astype(np.int32)
    w = rng.integers(1, 256, arcs).astype(np.uint32)
    g = b2.Graph.from_arrays(rp, ci, w)
    srv = Server(big_vertices=big_vertices)
    gid = srv.add_graph(g)
    assert srv.graph_config(gid)["cluster_team"] == cluster
    sources = [17, 0, int(ci[5])]
    outs = [srv.result_buffer(g) for _ in sources]
    for s, o in zip(sources, outs):
        srv.submit(gid, s, o)
    srv.progress(wait_all=True)
    assert [c["status"] for c in srv.poll()] == [0] * len(sources)
    for s, o in zip(sources, outs):
        assert np.array_equal(o.numpy().view(np.uint32), orc.dijkstra(rp, ci, w, s))
    srv.close()
    g.close()

"""GPU solves on several threads, graphs and streams at once: every one is right, and a small
graph's solve leaves room for others while two or more are under way."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["bf", "delta"])
def test_small_solves_share_the_device(b2, cuda, method):
    """Two solves are held in their progress callbacks while a third one is launched."""
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    hs = [b2.gen_er(3000, 24000, 1, 100, k) for k in range(3)]
    graphs = [b2.Graph.from_host(h, "u32") for h in hs]
    grid = lambda k: graphs[k].sssp(0, method=method)[2]["grid_blocks"]
    assert grid(0) == sms
    held, go = threading.Semaphore(0), threading.Event()
    failed = []

    def hold(k):
        first = []

        def progress(_):
            if not first:
                first.append(1)
                held.release()
                if not go.wait(60):
                    failed.append(k)
        try:
            graphs[k].sssp(0, method=method, stream=torch.cuda.Stream(), progress=progress)
        except Exception as e:   # noqa: BLE001
            failed.append(e)
            held.release()

    threads = [threading.Thread(target=hold, args=(k,)) for k in range(2)]
    try:
        threads[0].start()
        assert held.acquire(timeout=60)
        assert grid(2) == sms                     # two whole grids fit
        threads[1].start()
        assert held.acquire(timeout=60)
        assert grid(2) == sms // 4
        assert graphs[2].sssp(0, method=method, grid_blocks=100)[2]["grid_blocks"] == 100
    finally:
        go.set()
        for t in threads:
            if t.ident:
                t.join()
    assert not failed and grid(2) == sms
    big = b2.Graph.from_host(b2.gen_er(sms * 512 + 1, 4 * sms * 512, 1, 100, 0), "u32")
    assert big.sssp(0, method=method)[2]["grid_blocks"] > sms // 4
    for g in graphs + [big]:
        g.close()


def test_threads_with_graphs_of_their_own(b2, orc, cuda):
    torch = cuda
    hs = [b2.gen_er(500 * (k + 1), 3000 * (k + 1), 1, 100, k) for k in range(11)] + [b2.gen_er(90000, 500000, 1, 100, 3)]
    refs = [[orc.dijkstra(h.rowptr, h.colind, h.weights, s) for s in range(3)] for h in hs]
    graphs = [b2.Graph.from_host(h, "u32") for h in hs]
    wrong = []

    def work(k):
        try:
            stream = torch.cuda.Stream()
            for rep in range(24):
                s, method = rep % 3, ("bf", "delta", "bf", "adds")[rep % 4]
                out = torch.empty(graphs[k].n, dtype=torch.int32, device="cuda")
                stream.wait_stream(torch.cuda.default_stream())
                graphs[k].sssp(s, method=method, out=out, stream=stream, pred=bool(rep & 4))
                if not np.array_equal(out.cpu().numpy().view(np.uint32), refs[k][s]):
                    wrong.append((k, rep))
        except Exception as e:   # noqa: BLE001
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(hs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
    for g in graphs:
        g.close()

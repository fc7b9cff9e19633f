"""GPU solves that end early (a budget that runs out, a worklist that is too small): the
status and the bucket width they report, and the handle afterwards."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
POOL_EXHAUSTED, TIMEOUT = 4, 7


def _solve(b2, torch, g, out, **opts):
    o, st = b2.default_opts(**opts), b2._lib.Stats()
    rc = b2.lib().b2_sssp_delta(g._h, 0, C.c_void_p(out.data_ptr()), None, C.byref(o),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(st))
    return rc, st.as_dict()


# budgets from less than a barrier to a few phases: the wait that notices may be any block's
@pytest.mark.parametrize("weight", ["u32", "f32"])
def test_width_of_failed_solves(b2, orc, cuda, weight):
    torch = cuda
    h = b2.gen_grid(150, 150, seed=3)
    g = b2.Graph.from_host(h, weight)
    out = torch.empty(g.n, dtype=torch.int32 if weight == "u32" else torch.float32, device="cuda")
    rc, whole = _solve(b2, torch, g, out)
    assert rc == 0 and whole["delta_final"] > 0
    width = whole["delta_final"]
    for k in range(300):
        rc, st = _solve(b2, torch, g, out, timeout_ms=0.001 * (1 + k % 60))
        assert rc in (0, TIMEOUT) and st["delta_final"] == width
    for capacity in (1, 5, 20, 60):
        rc, st = _solve(b2, torch, g, out, worklist_capacity=capacity)
        assert rc == POOL_EXHAUSTED and st["delta_final"] == width
    rc, st = _solve(b2, torch, g, out)
    assert rc == 0
    ref = orc.dijkstra(h.rowptr, h.colind, h.weights if weight == "u32" else h.fweights, 0)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), np.ascontiguousarray(ref).view(np.uint32))
    g.close()

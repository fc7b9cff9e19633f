"""GPU scratch kept between calls: it is given back on request, and calls go on as before."""
import pytest

pytestmark = pytest.mark.gpu


def test_scratch_is_given_back(b2, cuda):
    torch = cuda
    n = 6000
    d0 = torch.full((n, n), float("inf"), device="cuda")
    d0[torch.arange(n - 1), torch.arange(1, n)] = 1.0
    d0.fill_diagonal_(0)
    small = d0[:300, :300].contiguous()
    want = small.clone()
    b2.apsp(want)
    # only this call's scratch counts: whatever earlier tests left is released first
    b2.release_scratch()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    d = d0[:4000, :4000].contiguous()
    torch.cuda.synchronize()
    free = min(free, torch.cuda.mem_get_info()[0])
    b2.apsp(d)
    torch.cuda.synchronize()
    kept = free - torch.cuda.mem_get_info()[0]
    assert kept >= 4000 * 4000 * 4
    b2.release_scratch()
    assert torch.cuda.mem_get_info()[0] >= free
    b2.release_scratch()   # (nothing left)
    b2.apsp(small)
    assert torch.equal(small, want)


def test_scratch_in_use_stays(b2, cuda):
    """A product planned but not yet filled keeps its scratch."""
    torch = cuda
    import ctypes as C
    from b200sssp.minplus import _csr_view
    k = 3000
    rp = torch.arange(k + 1, dtype=torch.int64, device="cuda") * 5
    ci = (torch.arange(5 * k, device="cuda") * 7919 % k).to(torch.int32)
    v = torch.arange(5 * k, device="cuda").to(torch.int32) % 100
    want = b2.minplus_spgemm((rp, ci, v, k), (rp, ci, v, k))
    view, plan, nnz = _csr_view(rp, ci, v, k), C.c_void_p(), C.c_int64()
    L = b2.lib()
    assert L.b2_minplus_spgemm_plan(C.byref(view), C.byref(view), None, C.byref(plan), C.byref(nnz)) == 0
    b2.release_scratch()
    out = [torch.empty_like(x) for x in want]
    assert nnz.value == want[1].numel()
    assert L.b2_minplus_spgemm_fill(plan, *(C.c_void_p(x.data_ptr()) for x in out), None) == 0
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want))

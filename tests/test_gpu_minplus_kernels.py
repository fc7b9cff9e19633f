"""GPU parity of every dense min-plus kernel that the size rule picks, with the picked kernel checked.

A product takes a minimum of sums that are each rounded once, so it is the same word for word in
any order of k, tile or split: no tolerance.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MISS = 1073741823
KERNELS = {"tma": "k_minplus_tma(", "128": "Tile<16, 16, 32>", "64": "Tile<8, 8, 16>"}


def _operand(rng, shape, dtype):
    if dtype == np.float32:
        a = rng.uniform(-1, 1, shape).astype(np.float32)
        a[rng.uniform(size=shape) < 0.4] = np.inf
    else:
        a = rng.integers(-1000, 1001, shape).astype(np.int32)
        a[rng.uniform(size=shape) < 0.4] = MISS
    return a


def _picked(torch, f):
    """f's kernels by the names above (f has run before: its one-time set-up is done); None where
    the profiler sees no kernels at all."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    return {k for k, name in KERNELS.items() if any(name in n for n in names)} if any("k_" in n for n in names) else None


def _padded(torch, x, pad):
    buf = torch.zeros((x.shape[0], x.shape[1] + pad), dtype=torch.from_numpy(x).dtype, device="cuda")
    buf[:, :x.shape[1]] = torch.from_numpy(x).cuda()
    return buf[:, :x.shape[1]]


# (M, N, K), paddings of A, B and C: TMA with a partial last k tile (even and odd), rows and columns
# that are no multiple of its tile, outputs whose rows start on 16 bytes or not; the 128-tile kernel
# with 16-byte and 4-byte copies of A and with k chunks that cross its end, whole and split over a
# cluster; the 64-tile kernel whole and split
@pytest.mark.parametrize("dtype,kernel,mnk,pads", [
    (np.int32, "tma", (1400, 1408, 1000), (0, 0, 0)),
    (np.int32, "tma", (1410, 1412, 1004), (0, 0, 0)),
    (np.int32, "tma", (1411, 1407, 1003), (1, 1, 0)),
    (np.int32, "tma", (1409, 1401, 1001), (3, 3, 3)),
    (np.int32, "tma", (1500, 1500, 1026), (2, 0, 1)),
    (np.int32, "128", (1411, 1408, 1003), (0, 0, 0)),
    (np.int32, "128", (1300, 1410, 50), (2, 0, 2)),
    (np.int32, "128", (130, 130, 4001), (3, 0, 0)),
    (np.int32, "128", (260, 260, 4000), (0, 1, 0)),
    (np.int32, "64", (700, 650, 129), (3, 2, 0)),
    (np.int32, "64", (520, 520, 4001), (3, 0, 0)),
    (np.float32, "128", (1400, 1408, 1000), (0, 0, 0)),
    (np.float32, "128", (1411, 1407, 1003), (1, 1, 0)),
    (np.float32, "128", (1411, 1407, 1001), (0, 0, 1)),
    (np.float32, "128", (1300, 1410, 50), (2, 0, 2)),
    (np.float32, "128", (130, 130, 4001), (3, 0, 0)),
    (np.float32, "128", (260, 260, 4002), (0, 1, 0)),
    (np.float32, "64", (700, 650, 129), (3, 2, 0)),
    (np.float32, "64", (520, 520, 4001), (3, 0, 0))])
def test_every_kernel(b2, orc, cuda, dtype, kernel, mnk, pads):
    torch = cuda
    M, N, K = mnk
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A, B = _operand(rng, (M, K), dtype), _operand(rng, (K, N), dtype)
    a, b = _padded(torch, A, pads[0]), _padded(torch, B, pads[1])
    out = torch.full((M, N + pads[2]), 7, dtype=a.dtype, device="cuda")
    f = lambda: b2.minplus_gemm(a, b, out=out[:, :N])
    f()
    assert _picked(torch, f) in (None, {kernel})
    got = out.cpu().numpy()
    assert (got[:, N:] == 7).all()
    rows = np.unique(np.concatenate([np.arange(0, M, max(1, M // 300)), [M - 1], np.arange(120, min(M, 136))]))
    assert np.array_equal(got[rows, :N], orc.minplus_gemm(np.ascontiguousarray(A[rows]), B))


# all pairs by TMA products: a chain needs every squaring, shortcuts end it early (the products
# queued after that must leave the matrix alone)
@pytest.mark.parametrize("n,reach", [(1500, 1), (1500, 40), (1536, 7), (1408, 300)])
def test_all_pairs_by_tma(b2, orc, cuda, n, reach):
    torch = cuda
    rng = np.random.default_rng(n + reach)
    D = np.full((n, n), MISS, np.int32)
    D[np.arange(n - 1), np.arange(1, n)] = 1
    for k in range(2, reach):   # arcs further along the chain at no gain: fewer hops, the same distances
        D[np.arange(n - k), np.arange(k, n)] = k
    np.fill_diagonal(D, 0)
    keep = torch.from_numpy(D).cuda()
    d = keep.clone()
    count = b2.apsp(d)
    limit = int(np.ceil(np.log2(n - 1)))
    assert count == min(limit, int(np.ceil(np.log2((n - 1) / max(1, reach - 1)))) + 1)
    i = np.arange(n)
    want = np.where(i[None] >= i[:, None], i[None] - i[:, None], MISS).astype(np.int32)
    assert np.array_equal(d.cpu().numpy(), want)
    d.copy_(keep)
    picked = _picked(torch, lambda: b2.apsp(d))
    assert picked is None or "tma" in picked

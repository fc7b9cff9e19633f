"""GPU parity of the dense min-plus kernels at the edges of their tiles and splits.

The product takes a minimum of sums that are each rounded once, so it is the
same word for word in any order of k, tile or split: no tolerance.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MISS = 1073741823


def _operand(rng, shape, dtype):
    if dtype == np.float32:
        a = rng.uniform(-1, 1, shape).astype(np.float32)
        a[rng.uniform(size=shape) < 0.4] = np.inf
    else:
        a = rng.integers(-1000, 1001, shape).astype(np.int32)
        a[rng.uniform(size=shape) < 0.4] = MISS
    return a


# (M, N, K): one element; tile edges +- 1 of the 64 and 128 tiles; k tiles of
# 16 / 32 and their remainders; long k on few tiles (clusters of 2, 4 and 8
# blocks, uneven parts); wide and tall outputs; enough tiles for the unsplit
# kernels (the last one is whole 128-tiles: TMA for int32)
@pytest.mark.parametrize("dtype", [np.float32, np.int32])
@pytest.mark.parametrize("mnk", [(1, 1, 1), (63, 65, 15), (64, 64, 16), (65, 63, 17), (1, 300, 33), (300, 1, 31),
                                 (127, 129, 32), (64, 64, 1000), (33, 70, 2049), (128, 130, 515), (257, 255, 300),
                                 (500, 90, 700), (90, 500, 701), (700, 650, 129), (1400, 1500, 40),
                                 (1664, 1536, 36)])
def test_gemm_shapes(b2, orc, cuda, dtype, mnk):
    torch = cuda
    M, N, K = mnk
    rng = np.random.default_rng(M * 31 + N * 7 + K)
    A, B = _operand(rng, (M, K), dtype), _operand(rng, (K, N), dtype)
    C = b2.minplus_gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()).cpu().numpy()
    assert np.array_equal(C, orc.minplus_gemm(A, B))


# leading dimensions and bases that allow 16-, 8- or only 4-byte accesses, for
# a split product and for an unsplit one; the output's padding stays untouched
@pytest.mark.parametrize("dtype", [np.float32, np.int32])
@pytest.mark.parametrize("mnk", [(70, 140, 400), (1300, 1410, 50)])
@pytest.mark.parametrize("pads", [(0, 0, 0, 0), (4, 8, 12, 4), (2, 6, 2, 2), (1, 3, 5, 1), (8, 1, 4, 0), (3, 4, 0, 4)])
def test_gemm_alignment(b2, orc, cuda, dtype, mnk, pads):
    torch = cuda
    M, N, K = mnk
    pa, pb, pc, off = pads
    rng = np.random.default_rng(M + 17 * pa + 5 * pb + pc)
    A, B = _operand(rng, (M, K), dtype), _operand(rng, (K, N), dtype)

    def placed(x, pad):
        buf = torch.empty(x.shape[0] * (x.shape[1] + pad) + off, dtype=torch.from_numpy(x).dtype, device="cuda")
        view = buf[off:].view(x.shape[0], x.shape[1] + pad)
        view[:, :x.shape[1]] = torch.from_numpy(x).cuda()
        return view[:, :x.shape[1]]

    out = torch.full((M * (N + pc) + off,), 7, dtype=torch.from_numpy(A).dtype, device="cuda")
    C = out[off:].view(M, N + pc)
    b2.minplus_gemm(placed(A, pa), placed(B, pb), out=C[:, :N])
    got = C.cpu().numpy()
    assert np.array_equal(got[:, :N], orc.minplus_gemm(A, B))
    assert (got[:, N:] == 7).all() and (out[:off].cpu().numpy() == 7).all()


def test_gemm_split_nan_inf(b2, orc, cuda):
    """NaN candidates lose and -inf wins in a product whose k is split over a cluster."""
    torch = cuda
    rng = np.random.default_rng(5)
    A, B = _operand(rng, (60, 900), np.float32), _operand(rng, (900, 61), np.float32)
    A[rng.uniform(size=A.shape) < 0.2] = np.nan
    B[rng.uniform(size=B.shape) < 0.01] = -np.inf
    B[:, 7] = np.nan
    C = b2.minplus_gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()).cpu().numpy()
    R = orc.minplus_gemm(A, B)
    assert np.isinf(C[:, 7]).all()
    assert np.array_equal(np.isnan(C), np.isnan(R)) and np.array_equal(C[~np.isnan(R)], R[~np.isnan(R)])


# chains need every squaring (odd and even counts: the result ends in either
# buffer); a star is done after one and a complete graph changes nothing in the
# second, so the queued products after that must leave the matrix alone
@pytest.mark.parametrize("dtype", [np.float32, np.int32])
@pytest.mark.parametrize("kind,n", [("chain", 9), ("chain", 17), ("chain", 130), ("chain", 300), ("star", 40),
                                    ("star", 150), ("random", 65), ("random", 259), ("chain", 3)])
def test_apsp_stops_on_the_device(b2, orc, cuda, dtype, kind, n):
    torch = cuda
    rng = np.random.default_rng(n)
    miss = np.inf if dtype == np.float32 else MISS
    D = np.full((n, n), miss, dtype)
    if kind == "chain":
        D[np.arange(n - 1), np.arange(1, n)] = 1
    elif kind == "star":
        D[0, 1:] = 2
        D[1:, 0] = 3
    else:
        D[:] = rng.integers(1, 100, (n, n)).astype(dtype)
    np.fill_diagonal(D, 0)
    ref, count, limit = D.copy(), 0, int(np.ceil(np.log2(max(n - 1, 1))))
    while count < limit:
        nxt = orc.minplus_gemm(ref, ref)
        count += 1
        same = np.array_equal(nxt, ref)
        ref = nxt
        if same:
            break
    got = torch.from_numpy(D).cuda()
    assert b2.apsp(got) == count
    assert np.array_equal(got.cpu().numpy(), ref)

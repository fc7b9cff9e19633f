"""GPU parity of the SpGEMM row kernels at the edges of their row classes, bit for bit.

Every candidate is one rounded sum and a column's result is the smallest of
them, whatever the order, so the oracle's words are the only right ones.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MISS = 1073741823


def _values(rng, n, dtype):
    if dtype == np.float32:
        v = rng.uniform(-1, 1, n).astype(np.float32)
        v[rng.uniform(size=n) < 0.03] = np.inf
        v[rng.uniform(size=n) < 0.02] = np.nan
    else:
        v = rng.integers(-1000, 1000, n).astype(np.int32)
        v[rng.uniform(size=n) < 0.05] = MISS
    return v


def _check(b2, orc, torch, rows, blen, N, dtype, seed):
    """rows: column lists of A; blen: lengths of B's rows."""
    rng = np.random.default_rng(seed)
    K = len(blen)
    arp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    aci = np.concatenate(rows).astype(np.int32) if arp[-1] else np.zeros(0, np.int32)
    brp = np.concatenate([[0], np.cumsum(blen)]).astype(np.int64)
    bci = rng.integers(0, N, int(brp[-1])).astype(np.int32)
    A = (arp, aci, _values(rng, aci.size, dtype))
    B = (brp, bci, _values(rng, bci.size, dtype))
    cu = [tuple(torch.from_numpy(x).cuda() for x in m) for m in (A, B)]
    got = b2.minplus_spgemm((*cu[0], K), (*cu[1], N))
    ref = orc.minplus_spgemm(A, B, N)
    for g, r in zip(got, ref):
        assert np.array_equal(g.cpu().numpy().view(np.uint32), np.ascontiguousarray(r).view(np.uint32))


# columns: few (long runs of one column), many, and past the widths at which the
# column and the slot still share 32 bits (2^23 for whole warps, 2^25 for halves)
@pytest.mark.parametrize("dtype", [np.float32, np.int32])
@pytest.mark.parametrize("N", [1, 5, 40, 3000, (1 << 23) - 1, 1 << 23, (1 << 25) - 1, 1 << 25])
def test_rows_of_every_length(b2, orc, cuda, dtype, N):
    rng = np.random.default_rng(N % 1000)
    sizes = [0, 1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 112, 113, 127, 128, 129, 160, 192, 193,
             255, 256, 257, 384, 385, 511, 512, 513, 900]
    K = 400
    blen = np.ones(K, int)
    blen[100:200] = 0          # empty rows of B between others
    blen[200:300] = rng.integers(2, 12, 100)
    blen[300:] = 130
    rows = []
    for n in sizes:
        rows.append(rng.integers(0, 100, n))                     # many entries of one candidate each
        mixed, left = [], n                                      # few entries, gaps among them
        while left > 0:
            k = int(rng.integers(0, K))
            if blen[k] <= left:
                mixed.append(k)
                left -= blen[k]
        rows.append(np.array(mixed, int))
        rows.append(np.array([320] * (n // 130), int))           # nothing but long rows of B
    _check(b2, orc, cuda, rows, blen, N, dtype, N % 77)


# long rows: one pass of 49152 columns, its edges, several passes (where some of the
# rows are too short for them and are sorted), and the widest matrix that is
# accumulated densely and the first that is not
@pytest.mark.parametrize("dtype", [np.float32, np.int32])
@pytest.mark.parametrize("N", [3, 513, 1000, 24576, 24577, 49151, 49152, 49153, 130000, 196608, 196609, 786432,
                               786433])
def test_long_rows(b2, orc, cuda, dtype, N):
    rng = np.random.default_rng(N % 991)
    K = 1500
    blen = rng.integers(0, 60, K)
    blen[7] = 40000
    rows = [rng.integers(0, K, n) for n in (30, 511, 512, 513, 1024, 1025, 3000, 17)]
    rows += [np.array([7]), np.array([], int), np.array([7] * 3 + [9, 11])]
    _check(b2, orc, cuda, rows, blen, N, dtype, N % 83)


def test_long_row_bad_column(b2, cuda):
    """A column index out of range is reported from long rows too, also where A's entry is absent."""
    torch = cuda
    rp = torch.tensor([0, 600], dtype=torch.int64, device="cuda")
    ci = torch.zeros(600, dtype=torch.int32, device="cuda")
    ci[599] = 1
    v = torch.ones(600, dtype=torch.float32, device="cuda")
    v[599] = float("inf")
    brp = torch.tensor([0, 1, 2], dtype=torch.int64, device="cuda")
    bci = torch.tensor([0, 9], dtype=torch.int32, device="cuda")
    with pytest.raises(b2.B2Error) as e:
        b2.minplus_spgemm((rp, ci, v, 2), (brp, bci, torch.ones(2, device="cuda"), 2))
    assert e.value.status == 9

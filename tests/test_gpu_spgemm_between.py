"""GPU rows of wide sparse products that are sorted or accumulated densely by how many there are:
both ways and the lines between them give the oracle's words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MISS = 1073741823


# columns for two, four and sixteen passes; rows on both sides of 640 candidates a pass and of
# the most that is sorted (5120 below four passes, 8192 at four, at most 20000); a few rows
# (accumulated densely), at least 512 between the lines (sorted), and a few among many short
# ones, some of them sorted all the same (split off for dense accumulation)
@pytest.mark.parametrize("columns,passes", [(60000, 2), (196608, 4), (786432, 16)])
@pytest.mark.parametrize("kind", ["few", "many", "among"])
@pytest.mark.parametrize("dtype", [np.float32, np.int32])
def test_rows_between(b2, orc, cuda, columns, passes, kind, dtype):
    torch = cuda
    rng = np.random.default_rng(passes + len(kind))
    low, high = 640 * passes, 5120 if passes < 4 else min(20000, 8192 + 5800 * (passes - 4))
    lengths = [low - 1, low, low + 1, high - 1, high, high + 1, 7, 400, 0]
    if kind == "many":
        lengths = [low] * 400 + [low + 3] * 200 + lengths
    elif kind == "among":
        lengths = [3] * 600 + [600] * 5 + lengths
    K = 3000
    # row k of B has k % 40 entries; a row of A takes whole rows of B until its length is reached
    blen = np.arange(K) % 40
    rows = []
    for n in lengths:
        k, left = [], n
        while left > 0:
            c = int(rng.integers(0, K))
            if blen[c] <= left:
                k.append(c)
                left -= blen[c]
        rows.append(k)
    arp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    aci = np.concatenate([np.array(r, np.int32) for r in rows])
    brp = np.concatenate([[0], np.cumsum(blen)]).astype(np.int64)
    bci = rng.integers(0, columns, int(brp[-1])).astype(np.int32)

    def values(n):
        if dtype == np.float32:
            v = rng.uniform(-1, 1, n).astype(np.float32)
            v[rng.uniform(size=n) < 0.02] = np.inf
            v[rng.uniform(size=n) < 0.02] = np.nan
        else:
            v = rng.integers(-1000, 1000, n).astype(np.int32)
            v[rng.uniform(size=n) < 0.04] = MISS
        return v

    A, B = (arp, aci, values(aci.size)), (brp, bci, values(bci.size))
    cu = [tuple(torch.from_numpy(x).cuda() for x in m) for m in (A, B)]
    got = b2.minplus_spgemm((*cu[0], K), (*cu[1], columns))
    ref = orc.minplus_spgemm(A, B, columns)
    for g, r in zip(got, ref):
        assert np.array_equal(g.cpu().numpy().view(np.uint32), np.ascontiguousarray(r).view(np.uint32))

"""GPU sparse products whose columns meet zeros of both signs: the results are equal numbers, in every
class of rows (which of the zeros a column returns is not defined)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows of half a warp, of a warp, long ones in one pass over the columns, in several, and sorted
@pytest.mark.parametrize("columns", [40, 60000, 900000])
def test_zeros_of_both_signs(b2, orc, cuda, columns):
    torch = cuda
    rng = np.random.default_rng(columns)
    K = 500
    blen = rng.integers(1, 30, K)
    rows = [rng.integers(0, K, n) for n in (1, 3, 9, 20, 30, 90, 200, 400)]
    arp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    brp = np.concatenate([[0], np.cumsum(blen)]).astype(np.int64)
    bci = np.sort(rng.integers(0, columns, int(brp[-1]))).astype(np.int32) if columns > 40 else \
        rng.integers(0, columns, int(brp[-1])).astype(np.int32)
    zeros = np.array([0.0, -0.0, 0.0, -0.0, 1.0, -1.0, -np.inf], np.float32)
    A = (arp, np.concatenate(rows).astype(np.int32), rng.choice(zeros, int(arp[-1]), p=[.25, .35, .1, .1, .1, .09, .01]))
    B = (brp, bci, rng.choice(zeros, bci.size, p=[.25, .35, .1, .1, .15, .04, .01]))
    cu = [tuple(torch.from_numpy(x).cuda() for x in m) for m in (A, B)]
    rp, ci, v = (x.cpu().numpy() for x in b2.minplus_spgemm((*cu[0], K), (*cu[1], columns)))
    orp, oci, ov = orc.minplus_spgemm(A, B, columns)
    assert np.array_equal(rp, orp) and np.array_equal(ci, oci)
    assert np.array_equal(v, ov)

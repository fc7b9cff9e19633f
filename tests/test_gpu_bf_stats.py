"""GPU Bellman-Ford statistics: improvements count every lowered label, pushes each vertex once a round."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pred", [False, True])
def test_improvements_and_pushes(b2, cuda, pred):
    # 0 -> 2000 middle vertices -> 200 sinks, every sink at 2000 different distances.  A sink's
    # label is lowered more than once unless its smallest candidate comes first.
    middle, sinks = 2000, 200
    n = 1 + middle + sinks
    rng = np.random.default_rng(1)
    rp = np.concatenate([[0, middle], middle + sinks * np.arange(1, middle + 1), np.full(sinks, middle + sinks * middle)])
    ci = np.concatenate([np.arange(1, middle + 1), np.tile(np.arange(middle + 1, n), middle)])
    w = np.concatenate([np.ones(middle), np.argsort(rng.random((sinks, middle)), axis=1).T.ravel() + 1])
    g = b2.Graph.from_arrays(rp.astype(np.int64), ci.astype(np.int32), w.astype(np.uint32))
    d, _, st = g.sssp(0, method="bf", pred=pred)
    assert (d.cpu().numpy()[middle + 1:] == 2).all()
    assert st["pushes"] == middle + sinks
    assert middle + sinks < st["improvements"] <= st["edges_scanned"] == middle + sinks * middle
    g.close()

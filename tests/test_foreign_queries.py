"""Foreign queries (se_knn) that have no near neighbours to find, and the rules
by which queries are ordered and shared out, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _unsorted_max():
    """Most queries that are taken as given, one to a warp (60 warps per SM)."""
    import torch

    return 2 * (60 * torch.cuda.get_device_properties(0).multi_processor_count - 1)


def _tree(c, n, seed):
    rng = np.random.default_rng(seed)
    c.build(*rng.random((3, n)).astype(np.float32))
    return c.points(), rng


@pytest.mark.parametrize("k", [1, 9, 32])
@pytest.mark.parametrize("order", ["as given", "sorted"])
def test_nan_queries_are_not_searched(native, oracle, order, k):
    """A query with a NaN coordinate is near nothing: NaN distances, points of
    the tree, and no walk of the tree for it, alone or beside other queries."""
    m = 3_000 if order == "as given" else _unsorted_max() + 5_001
    with native.Context() as c:
        p, rng = _tree(c, 60_000, 5)
        q = rng.random((m, 3)).astype(np.float32)
        c.knn(q, k)
        plain = c.stats()
        bad = q.copy()
        bad[np.arange(m), np.arange(m) % 3] = np.nan
        bad[::5] = np.nan
        idx, d2 = c.knn(bad, k, with_d2=True)
        assert np.isnan(d2).all() and idx.min() >= 0 and idx.max() < len(p)
        assert c.stats()["nodes_visited"] == 0 and c.stats()["buckets_scanned"] == 0
        some = np.arange(m) % 7 == 3
        mixed = np.where(some[:, None], bad, q)
        idx, d2 = c.knn(mixed, k, with_d2=True)
        assert c.stats()["buckets_scanned"] <= plain["buckets_scanned"]
    assert np.isnan(d2[some]).all() and idx.min() >= 0 and idx.max() < len(p)
    check = np.flatnonzero(~some)[:: 1 + m // 4000]
    ei, ed = oracle.knn_exact(p, q[check], k)
    assert np.array_equal(idx[check], ei) and np.array_equal(d2[check], ed)

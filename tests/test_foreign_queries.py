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


@pytest.mark.parametrize("k", [1, 9, 32])
@pytest.mark.parametrize("order", ["as given", "sorted"])
def test_queries_whose_every_distance_overflows(native, oracle, order, k):
    """Queries so far away (or at infinity) that every squared distance is
    infinite: all points tie, the lowest indices win, and there is no walk."""
    m = 300 if order == "as given" else _unsorted_max() + 2_003
    far = np.float32([np.inf, -np.inf, 3e19, -3e19, 1e38, -3.4e38])
    with native.Context() as c:
        p, rng = _tree(c, 5_000, 6)
        q = rng.random((m, 3)).astype(np.float32)
        out = q.copy()
        out[np.arange(m), rng.integers(0, 3, m)] = far[rng.integers(0, len(far), m)]
        idx, d2 = c.knn(out, k, with_d2=True)
        assert c.stats()["nodes_visited"] == 0 and c.stats()["buckets_scanned"] == 0
        assert np.array_equal(idx, np.tile(np.arange(k, dtype=np.int32), (m, 1))) and np.isinf(d2).all()
        some = np.arange(m) % 9 == 4
        mixed = np.where(some[:, None], out, q)
        idx, d2 = c.knn(mixed, k, with_d2=True)
    ei, ed = oracle.knn_exact(p, mixed, k, brute=True)
    assert np.array_equal(idx, ei) and np.array_equal(d2, ed)


@pytest.mark.parametrize("k", [1, 9, 32])
def test_queries_some_of_whose_distances_overflow(native, oracle, k):
    """A tree so wide that a query's distances to some of its points overflow
    and to others do not."""
    rng = np.random.default_rng(7)
    x, y, z = (rng.random((3, 400)) * 2e19).astype(np.float32)
    with native.Context() as c:
        c.build(x, y, z)
        p = c.points()
        q = np.concatenate([p, (rng.random((200, 3)) * 6e19 - 2e19).astype(np.float32)])
        idx, d2 = c.knn(q, k, with_d2=True)
        ei, ed = oracle.knn_exact(p, q, k, brute=True)
        assert np.isinf(ed).any() and np.isfinite(ed).any()
        assert np.array_equal(idx, ei) and np.array_equal(d2, ed)
        assert np.array_equal(c.knn_self(k), oracle.knn_exact(p, p, k, brute=True)[0])


def test_small_tree_and_overflow(native, oracle):
    """Fewer points than neighbours: the first is repeated."""
    with native.Context() as c:
        c.build(*np.float32([[0.0, 1.0, 0.5], [0.0, 1.0, 0.25], [0.0, 1.0, 0.75]]))
        q = np.float32([[np.inf, 0, 0], [0.1, 0.1, 0.1]])
        idx, d2 = c.knn(q, 8, with_d2=True)
        ei, ed = oracle.knn_exact(c.points(), q, 8, brute=True)
    assert np.array_equal(idx, ei) and np.array_equal(d2, ed)

"""Foreign queries (se_knn) that have no near neighbours to find, and the rules
by which queries are ordered and shared out, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _unsorted_max(k):
    """Most queries that are taken as given, one to a warp."""
    return (180 if k <= 16 else 120) * _sms() - 1


def _tree(c, n, seed):
    rng = np.random.default_rng(seed)
    c.build(*rng.random((3, n)).astype(np.float32))
    return c.points(), rng


@pytest.mark.parametrize("k", [1, 9, 32])
@pytest.mark.parametrize("order", ["as given", "sorted"])
def test_nan_queries_are_not_searched(native, oracle, order, k):
    """A query with a NaN coordinate is near nothing: NaN distances, points of
    the tree, and no walk of the tree for it, alone or beside other queries."""
    m = 3_000 if order == "as given" else _unsorted_max(k) + 5_001
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
    m = 300 if order == "as given" else _unsorted_max(k) + 2_003
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


def _check(c, oracle, p, q, k, rows=4_000):
    idx, d2 = c.knn(q, k, with_d2=True)
    s = np.unique(np.r_[np.arange(min(len(q), 70)), np.arange(0, len(q), 1 + len(q) // rows), np.arange(len(q) - 70, len(q))])
    s = s[s >= 0]
    ei, ed = oracle.knn_exact(p, q[s], k)
    assert np.array_equal(d2[s], ed)
    assert np.array_equal(idx[s], ei)
    return c.profile()["query_launches"]


@pytest.mark.parametrize("k", [1, 8, 31])
def test_counts_on_both_sides_of_each_rule(native, oracle, k):
    """The last count taken as given and the first sorted one, counts on both
    sides of 4, 8, 16 and 32 queries to a warp, and both numbers of sort passes."""
    top = _unsorted_max(k)
    halvings = [40 * _sms() * per + d for per in (4, 8, 16, 32) for d in (-per, 1)]
    with native.Context() as c:
        p, rng = _tree(c, 30_000, 8)
        for n in [top, top + 1] + halvings:
            # alone, or with keys, their preparation, two passes and items
            assert _check(c, oracle, p, rng.random((n, 3)).astype(np.float32), k) == (6 if n > top else 1)
        if k == 8:
            assert _check(c, oracle, p, rng.random(((1 << 21), 3)).astype(np.float32), k) == 6
            assert _check(c, oracle, p, rng.random(((1 << 21) + 1, 3)).astype(np.float32), k) == 7


def _orders(p, rng, n):
    """Foreign queries in every kind of order: n of each."""
    u = len(p)
    near = (p[rng.integers(0, u, n)] + 0.003 * rng.standard_normal((n, 3))).astype(np.float32)
    tree = p[np.arange(n) * u // n] + np.float32(1e-5)
    one = np.repeat(p[u // 3: u // 3 + 1], n, 0)
    cluster = (p[u // 2] + 1e-3 * rng.standard_normal((n, 3))).astype(np.float32)
    part = near.copy()
    part[: n // 2 + 5] = cluster[: n // 2 + 5]
    part[n // 4: n // 4 + 40] = near[:40]
    holes = cluster.copy()
    holes[::3, 1] = np.nan
    return {"near": near, "tree": tree, "tree reversed": tree[::-1], "one point": one, "cluster": cluster,
            "two points": np.where((np.arange(n) % 2 == 0)[:, None], one, p[:1]), "part cluster": part,
            "outside": (rng.random((n, 3)) * 10 + 2).astype(np.float32), "cluster with NaN": holes}


@pytest.mark.parametrize("k", [1, 4, 10, 16, 24, 32])
@pytest.mark.parametrize("n", [2_999, 17_750, 20_011, 27_001, 60_007, 200_003])
def test_queries_close_together_and_in_order(native, oracle, n, k):
    """Queries that one warp takes in place of several, as given and sorted, and
    those that come in order already."""
    with native.Context() as c:
        p, rng = _tree(c, 50_000, 9)
        for name, q in _orders(p, rng, n).items():
            q = np.ascontiguousarray(q, np.float32)
            ok = np.isfinite(q).all(1)
            idx, d2 = c.knn(q, k, with_d2=True)
            s = np.arange(0, n, 1 + n // 1_500)
            s = np.unique(np.r_[s, np.arange(min(n, 66)), np.arange(n - 66, n)])
            ei, ed = oracle.knn_exact(p, q[s[ok[s]]], k)
            assert np.array_equal(d2[s[ok[s]]], ed), name
            assert np.array_equal(idx[s[ok[s]]], ei), name
            assert np.isnan(d2[~ok]).all() and idx.min() >= 0 and idx.max() < len(p), name


@pytest.mark.parametrize("k", [1, 8, 31])
def test_trees_of_few_points(native, oracle, k):
    """Both sides of the size up to which queries share warps as given."""
    with native.Context() as c:
        for u in (1, 2, 7, 33, 100, 255, 256, 257):
            p, rng = _tree(c, u, 10)
            assert len(p) == u
            for n in (1, 100, 5_000, 70_001):
                q = (rng.random((n, 3)) * 3 - 1).astype(np.float32)
                q[::17] = np.nan
                q[5::17] = np.inf
                idx, d2 = c.knn(q, k, with_d2=True)
                ok = ~np.isnan(q).any(1)
                ei, ed = oracle.knn_exact(p, q[ok], k, brute=True)
                assert np.array_equal(d2[ok], ed) and np.array_equal(idx[ok], ei), (u, n)
                assert np.isnan(d2[~ok]).all() and idx.min() >= 0 and idx.max() < u


def test_trees_of_few_points_share_warps(native):
    """100 points are four buckets, and two of 5000 queries or more share a warp
    (one to a warp scanned 20,000 buckets)."""
    with native.Context() as c:
        _, rng = _tree(c, 100, 10)
        c.knn(rng.random((5_000, 3)).astype(np.float32), 32)
        assert 0 < c.stats()["buckets_scanned"] <= 2_500 * 4

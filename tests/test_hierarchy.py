"""The search hierarchy (leaves of at most 32 points, 32-way nodes above) at
the sizes and shapes where its levels, leaves and walk change: exact
neighbour lists against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uniform(rng, n):
    return rng.random((n, 3))


def _chain(rng, n):
    # halving distances towards the corner: subtrees that shed one point per level
    p = np.ldexp(1.0, -(np.arange(n) % 20))[:, None] * np.ones(3)
    return p * (1.0 + 0.3 * rng.random((n, 3)))


def _far_pairs(rng, n):
    # two clusters at opposite corners and points strewn between: warps across the gap
    p = rng.random((n, 3))
    p[: n // 3] *= 1e-3
    p[n // 3: 2 * n // 3] = 1.0 - 1e-3 * p[n // 3: 2 * n // 3]
    return p


def _lattice(rng, n):
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3), -1).reshape(-1, 3)
    return rng.permutation(g)[:n] / 64.0


SHAPES = {"uniform": _uniform, "chain": _chain, "far_pairs": _far_pairs, "lattice": _lattice}


@pytest.mark.parametrize("bucket", [1, 7, 32, 96])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_lists_exact_on_every_level_count(native, oracle, shape, bucket):
    rng = np.random.default_rng(11)
    with native.Context(leaf_bucket=bucket, build_octree=False) as c:
        for n in (1, 2, 31, 32, 33, 63, 65, 1023, 1025, 33_000):
            x, y, z = np.ascontiguousarray(SHAPES[shape](rng, n).astype(np.float32).T)
            c.build(x, y, z)
            p = c.points()
            k = min(12, len(p))
            idx, d2 = c.knn_self(k, with_d2=True)
            ei, ed = oracle.knn_exact(p, p, k)
            assert np.array_equal(idx, ei), (shape, bucket, n)
            assert np.array_equal(d2, ed), (shape, bucket, n)


def _shell(scale=2097151):
    """Integer points at one exact distance from a centre, as many as there
    are, and a few nearer ones: coordinates that the 21-bit code round trip
    keeps, corner points that pin the range."""
    f = np.float32
    v = np.arange(0, 400).astype(f)
    code = np.floor(f(scale) * (v / f(scale))).astype(np.int64)
    back = (code.astype(f) / f(scale)).astype(np.float64) * scale
    kept = set(np.flatnonzero(back.astype(f) == v).tolist())
    c = np.array([200, 200, 200])
    r = np.arange(-40, 41)
    o = np.stack(np.meshgrid(r, r, r), -1).reshape(-1, 3)
    o = o[np.array([all(int(t) in kept for t in p) for p in c + o])]
    n2 = (o**2).sum(1)
    best = np.bincount(n2[(n2 > 500) & (n2 < 1500)]).argmax()
    pts = np.concatenate([c + o[n2 == best], c + o[(n2 > 0) & (n2 <= 3)], [c], [[0, 0, 0]], [[scale] * 3]])
    return pts.astype(np.float32), int((n2 == best).sum())


@pytest.mark.parametrize("k", [1, 8, 10, 16, 24, 30, 32])
def test_more_ties_at_the_bound_than_slots(native, oracle, k):
    pts, ties = _shell()
    assert ties > 60  # more than any list keeps slots for
    x, y, z = (np.ascontiguousarray(a) for a in pts.T)
    with native.Context() as c:
        c.build(x, y, z)
        p = c.points()
        idx, d2 = c.knn_self(k, with_d2=True)
        ei, ed = oracle.knn_exact(p, p, k)
        assert np.array_equal(d2, ed)
        assert np.array_equal(idx, ei)


def test_nan_queries_get_points_of_the_tree(native, oracle):
    rng = np.random.default_rng(3)
    x, y, z = rng.random((3, 5_000)).astype(np.float32)
    q = rng.random((100, 3)).astype(np.float32)
    q[::7, 1] = np.nan
    with native.Context() as c:
        c.build(x, y, z)
        idx, d2 = c.knn(q, 9, with_d2=True)
        p = c.points()
    assert idx.min() >= 0 and idx.max() < len(p)
    ok = np.isfinite(q).all(1)
    assert np.isnan(d2[~ok]).all()
    ei, ed = oracle.knn_exact(p, q[ok], 9)
    assert np.array_equal(idx[ok], ei) and np.array_equal(d2[ok], ed)


@pytest.mark.parametrize("n", [319, 740, 1_481, 2_959, 3_001, 11_840, 11_841, 23_681])
def test_few_queries_per_warp(native, oracle, n):
    """Counts on both sides of each halving of the queries per warp."""
    rng = np.random.default_rng(n)
    x, y, z = rng.random((3, n)).astype(np.float32)
    with native.Context(build_octree=False) as c:
        c.build(x, y, z)
        p = c.points()
        assert np.array_equal(c.knn_self(16), oracle.knn_exact(p, p, 16)[0])
        assert np.array_equal(c.knn_self(16, 5, 301), oracle.knn_exact(p, p[5:306], 16)[0])


@pytest.mark.parametrize("k", [1, 8, 16, 31])
@pytest.mark.parametrize("shape", ["uniform", "far_pairs"])
def test_foreign_queries_in_any_order(native, oracle, shape, k):
    """Counts on both sides of the rule that sorts them; queries inside, on and
    far outside the tree's cube, and repeated ones; host and device memory."""
    import torch

    rng = np.random.default_rng(17)
    x, y, z = np.ascontiguousarray(SHAPES[shape](rng, 40_000).astype(np.float32).T)
    with native.Context() as c:
        c.build(x, y, z)
        p = c.points()
        for n in (1, 33, 3_000, 17_759, 17_761, 40_001):
            q = rng.random((n, 3)).astype(np.float32)
            q[::5] = p[rng.integers(0, len(p), len(q[::5]))]
            q[::11] = q[0]
            q[::13] *= 3.0
            ei, ed = oracle.knn_exact(p, q, k)
            idx, d2 = c.knn(q, k, with_d2=True)
            assert np.array_equal(idx, ei) and np.array_equal(d2, ed), n
            ti = c.knn(torch.from_numpy(q).cuda(), k)
            assert np.array_equal(ti.cpu().numpy(), ei), n


@pytest.mark.parametrize("k", [1, 2, 16, 32])
def test_compat_search_at_thread_counts(native, oracle, k):
    """The reference's search on counts around a warp and a block, and on more
    queries than there are threads at once (threads take several)."""
    rng = np.random.default_rng(23)
    x, y, z = rng.random((3, 90_000)).astype(np.float32)
    with native.Context(search_compat=True) as c:
        c.build(x, y, z)
        p, nodes = c.points(), c.octree()
        for start, n in ((0, 1), (7, 31), (100, 33), (0, 64), (5, 65), (3, 1_000)):
            assert np.array_equal(c.knn_self(k, start, n), oracle.knn_compat(nodes, p, p[start:start + n], k))
        idx = c.knn_self(k)
        s = slice(0, len(p), 37)
        assert np.array_equal(idx[s], oracle.knn_compat(nodes, p, p[s], k))

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

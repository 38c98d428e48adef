"""Searches of the tree's own points whose work items are listed first, cut at
Morton jumps, against the oracle, on both sides of the rules for the list and
for the points per warp."""
import numpy as np
import pytest

from shapeextraction_b200 import synth

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _cloud(kind, n, rng):
    if kind == "scene":
        return synth.scene(n, int(rng.integers(1000)))
    if kind == "jumps":  # small clumps all over the cube: every few points a jump
        c = rng.random((n // 9 + 1, 3))
        return (np.repeat(c, 9, 0)[:n] + 1e-4 * rng.standard_normal((n, 3))).T
    if kind == "line":
        t = rng.random(n)
        return np.stack([t, t, t])
    if kind == "plane":
        return np.stack([rng.random(n), rng.random(n), np.full(n, 0.5)])
    g = rng.integers(0, 70, (n, 3))  # equal distances, equal prefixes, equal points
    return g.T / 64.0


def _check(c, oracle, k, rng, start=0, count=None):
    p = c.points()
    count = len(p) - start if count is None else count
    idx, d2 = c.knn_self(k, start, count, with_d2=True)
    s = np.unique(np.r_[0:min(count, 80), rng.integers(0, count, 3_000), max(0, count - 80):count])
    ei, ed = oracle.knn_exact(p, p[start + s], k)
    assert np.array_equal(idx[s], ei) and np.array_equal(d2[s], ed)
    launches = c.profile()["query_launches"]
    per_warp = c.normals(k, start, count)
    assert np.isfinite(per_warp).all()
    return launches


@pytest.mark.parametrize("kind", ["scene", "jumps", "line", "plane", "grid"])
@pytest.mark.parametrize("k", [1, 8, 10, 16, 24, 32])
def test_listed_searches_are_exact(native, oracle, kind, k):
    rng = np.random.default_rng(31)
    with native.Context(build_octree=False) as c:
        for n in (12_001, 25_003, 50_017, 90_001, 200_003):
            x, y, z = (np.ascontiguousarray(v, np.float32) for v in _cloud(kind, n, rng))
            c.build(x, y, z)
            _check(c, oracle, k, rng)


def test_both_sides_of_the_rules(native, oracle):
    """One launch without the list, two with it; part of a tree, 30-bit codes."""
    rng = np.random.default_rng(32)
    sms = _sms()
    with native.Context(build_octree=False) as c, native.Context(code_bits=30, build_octree=False) as c30:
        x, y, z = (np.ascontiguousarray(v, np.float32) for v in rng.random((3, 2600 * sms + 4_000)))
        u = c.build(x, y, z)["n_points"]
        for k, most in ((8, 2600), (12, 1500), (24, 750)):
            for count, launches in ((40 * sms, 1), (80 * sms - 8, 1), (80 * sms, 2), (min(most, 1600) * sms, 2),
                                    (most * sms, 2), (most * sms + 1, 1)):
                assert _check(c, oracle, k, rng, int(rng.integers(0, u - count)), count) == launches, count
        c30.build(x[:100_000], y[:100_000], z[:100_000])
        assert _check(c30, oracle, 16, rng) == 2


@pytest.mark.parametrize("kind,more", [("line", 1.5), ("plane", 1.5)])
def test_few_cuts_without_jumps(native, kind, more):
    """Along a line and on a plane most neighbours in the Morton order are
    neighbours: the cuts add few node visits to those of whole warps. (Judged by
    the codes alone a line is cut into four times as many parts.)"""
    rng = np.random.default_rng(33)
    most = 750 * _sms()  # points of a listed search with k > 16
    with native.Context(build_octree=False) as c:
        u = c.build(*(np.ascontiguousarray(v, np.float32) for v in _cloud(kind, most + 9_000, rng)))["n_points"]
        assert u > most
        nodes = []
        for count, launches in ((most, 2), (most + 1, 1)):
            c.knn_self(24, 0, count)
            assert c.profile()["query_launches"] == launches
            nodes.append(c.stats()["nodes_visited"])
    assert nodes[0] < more * nodes[1], nodes


def test_listed_searches_leave_the_tree_as_it_was(native):
    """The list lives in the build's scratch: the tree, another search and
    another build come out the same."""
    x, y, z = synth.scene(60_000, 4)
    with native.Context() as c, native.Context() as other:
        for n in (60_000, 3_000, 20_000, 60_000):
            c.build(x[:n], y[:n], z[:n])
            other.build(x[:n], y[:n], z[:n])
            a = c.knn_self(16)
            b = c.normals(8)
            assert np.array_equal(a, c.knn_self(16)) and np.array_equal(b, c.normals(8))
            assert c.octree().tobytes() == other.octree().tobytes()
            assert np.array_equal(c.codes(), other.codes())
            assert np.array_equal(a, other.knn_self(16))

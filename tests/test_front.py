"""The one-block front of a small build (at most 8192 points) against the
oracle, bit for bit, on both sides of each of its sizes, and its errors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 31, 33, 1023, 1024, 1025, 2048, 2049, 4095, 4097, 8191, 8192, 8193]


def _cloud(kind, n):
    rng = np.random.default_rng(n)
    if kind == "uniform":
        p = rng.random((n, 3))
    elif kind == "repeats":  # many equal codes, and digits that all keys share
        p = rng.integers(0, 6, (n, 3)) / 8.0
    else:  # negative coordinates, a wide range
        p = rng.normal(0.0, 1e3, (n, 3))
    return np.ascontiguousarray(p.astype(np.float32).T)


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("kind", ["uniform", "repeats", "wide"])
def test_small_builds_bit_exact(native, oracle, kind, bits):
    with native.Context(code_bits=bits, root_compat=False) as c:
        for n in SIZES:
            x, y, z = _cloud(kind, n)
            info = c.build(x, y, z)
            ref = oracle.build_stages(x, y, z, code_bits=bits, root_compat=False)
            assert np.array_equal(c.codes(), ref["codes"]), (kind, bits, n)
            assert c.points().tobytes() == np.asarray(ref["points"], np.float32).tobytes(), (kind, bits, n)
            assert (info["min_coord"], info["max_coord"]) == (ref["min"], ref["max"])
            if info["n_points"] < 3:
                continue
            r = c.radix()
            for key in ("leftChild", "prefixN", "hasLeafLeft", "hasLeafRight", "parent"):
                assert np.array_equal(r[key], ref["radix"][key][: len(r[key])]), (key, kind, bits, n)
            assert c.octree().tobytes() == ref["octree"]["nodes"].tobytes(), (kind, bits, n)


@pytest.mark.parametrize("n", [5, 3_000, 8_192])
def test_small_builds_reject_nonfinite(native, n):
    x, y, z = _cloud("uniform", n)
    with native.Context() as c:
        for bad in (np.nan, np.inf, -np.inf):
            w = y.copy()
            w[n // 2] = bad
            with pytest.raises(native.ShapexError) as e:
                c.build(x, w, z)
            assert e.value.status == 5  # SE_ERR_NONFINITE
        c.build(x, y, z)
        assert c.profile()["build_ms"]["total"] > 0.0

"""Which clouds of a batch are queried on their build lane and which in the
launches shared per k, and that every cloud equals its single-cloud call on
both, in pinned host and device memory, through plain launches and the graph."""
import numpy as np
import pytest

from shapeextraction_b200 import synth

pytestmark = pytest.mark.gpu


def _batch(sizes):
    clouds = [synth.scene(s, seed=700 + i) if s > 0 else (np.zeros(0, np.float32),) * 3 for i, s in enumerate(sizes)]
    offsets = np.zeros(len(sizes) + 1, np.int64)
    offsets[1:] = np.cumsum(sizes)
    return clouds, offsets, [np.concatenate([cl[j] for cl in clouds]) for j in range(3)]


def _check(c, clouds, ks, offsets, xyz, pinned):
    import torch

    host = [torch.from_numpy(v) for v in xyz]
    arrays = tuple(h.pin_memory() if pinned else h.cuda() for h in host)
    out = torch.zeros((int(offsets[-1]), 3), dtype=torch.float32)
    out = out.pin_memory() if pinned else out.cuda()
    for _ in range(3):  # recorded, replayed
        out.zero_()
        _, _, u = c.normals_batch(arrays, (ks, offsets), out=out)
        launches = c.profile()["query_launches"]
    nrm = out.cpu().numpy()
    for i, (x, y, z) in enumerate(clouds):
        if x.size == 0:
            assert u[i] == 0
            continue
        c.build(x, y, z)
        assert u[i] == c.info()["n_points"]
        assert np.array_equal(nrm[offsets[i]:offsets[i] + u[i]], c.normals(int(ks[i]))), i
    return launches


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("graph", [True, False])
def test_lanes_by_size(native, graph, pinned):
    sizes = [150_000, 70_000, 3000, 500, 65_536, 65_535, 1, 0, 20_000, 900, 800]
    ks = np.array([16, 32, 8, 16, 10, 16, 8, 16, 5, 5, 5], np.int32)
    with native.Context(batch_graph=graph, batch_lane_min_points=65_536) as c:
        # three by their size; k = 16, 8, 5 are shared by two, two and three; the collecting launch
        clouds, offsets, xyz = _batch(sizes)
        assert _check(c, clouds, ks, offsets, xyz, pinned) == 3 + 3 + 1


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("graph", [True, False])
def test_lanes_by_sharing(native, graph, pinned):
    sizes = [3_000, 70_000, 65_536, 65_535, 66_000, 2_000, 2_001, 0, 70_000, 9_000, 800]
    ks = np.array([7, 16, 16, 10, 10, 24, 24, 24, 32, 32, 32], np.int32)
    with native.Context(batch_graph=graph) as c:
        clouds, offsets, xyz = _batch(sizes)
        # lanes: the only one of k = 7, both of k = 16, one of k = 10; launches for the rest of
        # k = 10 and for 24 (two small ones) and 32 (three); the collecting launch
        assert _check(c, clouds, ks, offsets, xyz, pinned) == 4 + 3 + 1


def test_a_k_of_its_own_per_cloud(native):
    ks = np.arange(1, 33, dtype=np.int32)
    with native.Context() as c:
        clouds, offsets, xyz = _batch([300 * k for k in range(1, 33)])
        assert _check(c, clouds, ks, offsets, xyz, False) == 32 + 1

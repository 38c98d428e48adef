"""Neighbour lists into every kind of output: aligned to 16 bytes or not (rows are
written 16 bytes at a time where they can be), device, pinned and pageable host
memory, the tree's own points and foreign ones in another order."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 7


def _buffers(where, n, k, offset):
    """Index and distance buffers that begin `offset` words past a 16-byte
    boundary, with guard words behind: (views, whole)."""
    import torch

    idx = torch.full((n * k + 8,), GUARD, dtype=torch.int32)
    d2 = torch.full((n * k + 8,), float(GUARD))
    if where == "pinned":
        idx, d2 = idx.pin_memory(), d2.pin_memory()
    elif where == "device":
        idx, d2 = idx.cuda(), d2.cuda()
    assert idx.data_ptr() % 16 == 0 and d2.data_ptr() % 16 == 0
    return [b[offset:offset + n * k].view(n, k) for b in (idx, d2)], [idx, d2]


@pytest.mark.parametrize("where", ["device", "pinned", "pageable"])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 10, 12, 16, 20, 24, 28, 32])
def test_lists_in_any_output(native, oracle, where, k):
    rng = np.random.default_rng(41)
    L = native.lib()
    with native.Context(build_octree=False) as c:
        c.build(*rng.random((3, 30_000)).astype(np.float32))
        p = c.points()
        q = rng.random((30_000, 3)).astype(np.float32)
        s = np.r_[0:40, 5_000:30_000:97, 29_960:30_000]
        own, foreign = oracle.knn_exact(p, p[s], k), oracle.knn_exact(p, q[s], k)
        for offset in (0, 1, 2, 4):
            (idx, d2), whole = _buffers(where, 30_000, k, offset)
            c.knn_self(k, out=idx, out_d2=d2, with_d2=True)
            assert np.array_equal(idx.cpu().numpy()[s], own[0]) and np.array_equal(d2.cpu().numpy()[s], own[1])
            (idx, d2), whole = _buffers(where, 30_000, k, offset)
            import torch

            queries = torch.from_numpy(q).cuda() if where == "device" else torch.from_numpy(q)
            rc = L.se_knn(c.handle, k, ctypes.c_void_p(queries.data_ptr()), len(q), ctypes.c_void_p(idx.data_ptr()),
                          ctypes.c_void_p(d2.data_ptr()), native.SE_MEM_DEVICE if where == "device" else native.SE_MEM_HOST)
            assert rc == 0
            assert np.array_equal(idx.cpu().numpy()[s], foreign[0]) and np.array_equal(d2.cpu().numpy()[s], foreign[1])
            for b in whole:  # nothing before or behind the rows
                b = b.cpu().numpy()
                assert (b[:offset] == GUARD).all() and (b[offset + 30_000 * k:] == GUARD).all()

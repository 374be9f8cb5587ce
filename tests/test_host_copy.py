"""Large copies between pageable arrays and the device (pinned ring, helper
threads): sizes at the pieces' and thresholds' edges, several contexts in
threads at once, and results that outlive their context."""
import gc
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from rustcolmap_b200 import MvsOptions, mvs

KB, MB = 1 << 10, 1 << 20
# pixels of a 3-channel image whose bytes lie at 256 KB, 1 MB, 3 MB, 6 MB, 24 MB
EDGES = [n // 3 + d for n in (256 * KB, MB, 3 * MB, 6 * MB, 24 * MB) for d in (0, 1)]


def round_trip(ctx, n, seed):
    rows = 1 if n < 8 * MB else 2  # a side is at most 2^23
    n = -(-n // rows)
    img = np.random.default_rng(seed).integers(0, 256, (rows, n, 3), dtype=np.uint8)
    _, rgb = mvs.resize_view(img, n, rows, ctx)  # the same size: the bytes themselves
    return np.array_equal(rgb, img)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1] + EDGES)
def test_gpu_copy_sizes(n):
    ctx = mvs.Context(0)
    assert round_trip(ctx, n, n) and round_trip(ctx, n, n + 1)
    ctx.close()


@pytest.mark.gpu
def test_gpu_copy_from_threads():
    def work(k):
        ctx = mvs.Context(0)
        ok = all(round_trip(ctx, n, 10 * k + i) for i, n in enumerate(EDGES[4:8]))
        ctx.close()
        return ok

    with ThreadPoolExecutor(7) as ex:  # more than there are rings
        assert all(ex.map(work, range(14)))


@pytest.mark.gpu
def test_gpu_results_outlive_context():
    ctx = mvs.Context(0)
    rng = np.random.default_rng(3)
    xyz = rng.uniform(-1, 1, (50000, 3))
    rgb = rng.integers(0, 256, (50000, 3)).astype(np.uint8)
    a, c = mvs.fuse_reduce(xyz, rgb, xyz, MvsOptions(voxel_rel=1e-6), ctx)
    first = a[:1].copy()
    ctx.close()
    del c
    gc.collect()
    b, _ = mvs.fuse_reduce(xyz, rgb, xyz, MvsOptions(voxel_rel=1e-6))
    assert len(a) == 50000 and np.array_equal(a, b) and np.array_equal(a[:1], first)
    a[0] = 7.0  # an ordinary array
    assert a.flags.writeable and b[0, 0] != 7.0

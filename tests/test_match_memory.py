"""Matching where the device has no room for the tensor-core search's packed
frames (as large as the descriptors): the FP32 kernels answer, as they did
when they were the only way, with the same matches."""
import contextlib

import numpy as np
import pytest

from rustcolmap_b200 import mvs, sift

pytestmark = pytest.mark.gpu

MB = 1 << 20
FRAMES, N = 40, 10000
DESC = FRAMES * N * 512  # bytes of the descriptors, and about of the packed frames


def _descs(wild):
    rng = np.random.default_rng(5)
    sets = [rng.random((N, 128), dtype=np.float32) for _ in range(2)]
    sets = [s / np.linalg.norm(s, axis=1, keepdims=True) for s in sets]
    sets[1][:3000] = sets[0][7000:] * (1 + 0.02 * rng.random((3000, 128), dtype=np.float32))
    if wild:
        sets[0][11, 5] = 3000.0  # past the packed range: both ways are tried
    sets += [sets[1]] * (FRAMES - 2)  # in no pair, but part of the call
    return [np.ascontiguousarray(s) for s in sets]


@pytest.mark.parametrize("wild,left", [(False, DESC + 150 * MB), (True, 2 * DESC + 60 * MB), (False, 2 * DESC + 60 * MB)])
def test_less_room_than_the_search_takes(wild, left):
    """Room for the descriptors, two pairs' tile partials (72 MB) and 70 MB
    more, or for the packed frames too but then not for the partials."""
    import torch
    sets, pairs = _descs(wild), [(0, 1), (1, 0)]
    with contextlib.closing(mvs.Context(0)) as ctx:
        want = sift.match_pairs(sets, pairs, 0.8, ctx)
        assert len(want[0][0]) >= 2900
    with contextlib.closing(mvs.Context(0)) as ctx:
        small = [s[:2100] for s in sets[:2]]
        sift.match_pairs(small, pairs, 0.8, ctx)  # every kernel is loaded
        sift.match_pairs([s[:300] for s in small], pairs, 0.8, ctx)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        hold = torch.empty(max(free - left, 0), dtype=torch.uint8, device="cuda")
        try:
            for _ in range(2):  # again: what the first call kept is in the way
                got = sift.match_pairs(sets, pairs, 0.8, ctx)
                for (a, b), (c, d) in zip(got, want):
                    assert np.array_equal(a, c) and np.array_equal(b, d)
        finally:
            del hold
            torch.cuda.empty_cache()

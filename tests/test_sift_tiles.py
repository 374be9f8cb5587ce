"""The SIFT octave kernel at the edges of its tiles (62 x 30 answered pixels of
64 x 32) against the CPU oracle, and the selection that stays on the device
(up to 8192 features) against the general path: the first features of a larger
request, bit for bit."""
import numpy as np
import pytest

from rustcolmap_b200 import mvs, sift

from test_sift import match, oracle_sift


def texture(h, w, seed):
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 256, (h // 3 + 2, w // 3 + 2)).astype(np.float64)
    a = np.repeat(np.repeat(a, 3, 0), 3, 1)[:h, :w]
    return a.astype(np.uint8)


@pytest.fixture(scope="module")
def ctx():
    c = mvs.Context(0)
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(62, 30), (63, 31), (64, 32), (65, 33), (124, 60), (125, 61), (126, 92), (187, 17),
                                 (40, 300), (641, 479)])
def test_gpu_sift_tile_edges(ctx, w, h):
    img = texture(h, w, w * 1000 + h)
    (op, od, oc, oraw), _ = oracle_sift(img)
    f = sift.extract_sift(img, ctx=ctx)
    assert f.n_raw == oraw and oraw > 0
    # libm's last bit may move a peak decision of 1% of the keypoints, or of one
    slack = max(1, len(op) // 100)
    assert abs(len(f.pts) - len(op)) <= slack
    assert (1.0 - match((f.pts, f.desc), (op, od))) * len(f.pts) <= slack


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [1, 63, 500, 2048, 8192, 8193])
@pytest.mark.parametrize("thr", [0.0067, 0.0])
def test_gpu_sift_first_features(ctx, cap, thr):
    img = texture(700, 1100, 5)
    img[200:330, 300:600] = 90  # flat: no keypoints there
    every = sift.extract_sift(img, opts=sift.SiftOptions(max_features=1000000, contrast_thr=thr), ctx=ctx)
    some = sift.extract_sift(img, opts=sift.SiftOptions(max_features=cap, contrast_thr=thr), ctx=ctx)
    n = min(cap, len(every.pts))
    assert len(every.pts) > 2048 and len(some.pts) == n and some.n_raw == every.n_raw
    assert np.array_equal(some.pts, every.pts[:n])
    assert np.array_equal(some.desc, every.desc[:n])
    assert np.array_equal(some.colors, every.colors[:n])

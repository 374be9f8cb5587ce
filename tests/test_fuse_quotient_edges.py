"""The device's quotients by a shared reciprocal at the edges of the exponents
they are formed for (numerators 2^-900 .. 2^900, divisors 2^-100 .. 2^100;
outside, zeros and subnormals are divided): poses, focal lengths, depths and
cells on both sides of each, against the oracle's divisions bit for bit."""
import contextlib

import numpy as np
import pytest

from oracle import oracle
from rustcolmap_b200 import MvsOptions, mvs
from rustcolmap_b200.types import Cam, ViewData

pytestmark = pytest.mark.gpu

W, H = 12, 9


def _views(n, f, t, cx=5.0, cy=4.0, k=0.0):
    rng = np.random.default_rng(3)
    return [ViewData(f"v{i}", i, W, H, Cam(f, cx, cy, k), np.eye(3), np.array(t, np.float64),
                     rng.integers(0, 256, (H, W)).astype(np.uint8), rng.integers(0, 256, (H, W, 3)).astype(np.uint8))
            for i in range(n)]


def _same(views, z, least):
    """Views of one pose and depth: every pixel's point is an average over
    all of them."""
    n = len(views)
    dms = [np.full((H, W), z, np.float32) for _ in views]
    order = [[j for j in range(n) if j != i] for i in range(n)]
    opts = MvsOptions(min_consistent=n - 1)
    off = np.cumsum([0] + [len(o) for o in order])
    want, wrgb, wper = oracle.fuse_candidates(views, dms, off, [x for o in order for x in o], list(range(n)), opts)
    assert len(want) >= least
    with contextlib.closing(mvs.Context(0)) as ctx:
        got, rgb, per = mvs.fuse_candidates(views, dms, order, list(range(n)), opts, ctx)
    assert np.array_equal(per, wper) and np.array_equal(rgb, wrgb)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("e", [-1074, -1030, -1022, -902, -901, -900, -899, -898, 0, 897, 898, 899, 900, 901, 1018])
@pytest.mark.parametrize("n", [2, 3, 6, 7])
def test_numerators(e, n):
    """The mean's numerator is about n 2^e: the pixel on the principal point
    has the camera centre's coordinates."""
    m = 1.0 + np.random.default_rng(n).random()
    _same(_views(n, 10.0, [np.ldexp(m, e), -np.ldexp(1.9 * m, e), 0.0]), 3.0, W)


@pytest.mark.parametrize("e", [-103, -101, -100, -99, 0, 98, 99, 100, 101, 120])
@pytest.mark.parametrize("k", [0.0, 1e-3])
def test_focal_lengths(e, k):
    if k and e < 0:
        k = np.ldexp(1e-3, 2 * e)  # the radius squared is about 2^-2e
    f = float(np.ldexp(1.37, e))
    _same(_views(3, f, [0.25, 0.0, -0.5], cx=4.3, cy=3.7, k=k), 2.5, W)


@pytest.mark.parametrize("e", [-3, 60, 97, 98, 99, 100, 101, 110])
def test_depths(e):
    _same(_views(4, 21.0, [0.0, 0.0, 0.0], cx=5.5, cy=3.25), np.float32(np.ldexp(1.61, e)), W)


@pytest.mark.parametrize("e", [-29, 0, 97, 98, 99, 100, 101, 300])
def test_cells(e):
    """Voxel keys of points around multiples of cells of both sides' sizes."""
    rng = np.random.default_rng(7)
    sparse = np.ldexp(np.array([[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]] * 50), e + 6)
    opts = MvsOptions(voxel_rel=2.0 ** -6 / np.sqrt(3.0))
    xyz = np.ldexp(rng.integers(-40, 41, (3000, 3)) * (1 + rng.integers(-2, 3, (3000, 3)) * 2.0 ** -52), e)
    rgb = rng.integers(0, 256, xyz.shape).astype(np.uint8)
    wx, wc = oracle.fuse_reduce(xyz, rgb, sparse, opts)
    with contextlib.closing(mvs.Context(0)) as ctx:
        gx, gc = mvs.fuse_reduce(xyz, rgb, sparse, opts, ctx)
    assert np.array_equal(gx, wx) and np.array_equal(gc, wc)

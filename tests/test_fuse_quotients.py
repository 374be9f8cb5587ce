"""Fusion's arithmetic shortcuts.  The quotient by a shared reciprocal
(y = 1 / b rounded, a y, two fused corrections) against division, and the
per-voxel sums of both lane groups against sequential numpy sums."""
import ctypes as C

import numpy as np
import pytest

from rustcolmap_b200 import MvsOptions, mvs

libm = C.CDLL("libm.so.6")
libm.fma.restype = C.c_double
libm.fma.argtypes = [C.c_double] * 3


def quot(a, b):
    y = 1.0 / b
    q = a * y
    q = libm.fma(libm.fma(-b, q, a), y, q)
    return libm.fma(libm.fma(-b, q, a), y, q)


@pytest.mark.parametrize("span", [1, 30, 90])
def test_quotient_by_reciprocal_is_the_division(span):
    rng = np.random.default_rng(span)
    n = 20000
    m = rng.integers(0, 2**52, (2, n), dtype=np.int64)
    # mantissas at the ends of the range, where the reciprocal rounds worst
    m[0, : n // 4] = 2**52 - 1 - rng.integers(0, 4, n // 4)
    m[1, n // 8 : n // 2] = rng.integers(0, 4, n // 2 - n // 8)
    m[1, n // 2 : 3 * n // 4] = 2**52 - 1 - rng.integers(0, 4, n // 4)
    e = rng.integers(-span, span + 1, (2, n))
    a, b = np.ldexp(1.0 + m * 2.0**-52, e)
    a *= rng.choice([-1.0, 1.0], n)
    got = np.array([quot(x, y) for x, y in zip(a.tolist(), b.tolist())])
    assert np.array_equal(got, a / b)


@pytest.fixture(scope="module")
def ctx():
    c = mvs.Context(0)
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(1, 1, 1), (1, 7, 8, 9), (3, 2, 15, 16, 17), (31, 32, 33, 5), (64, 65, 1, 700),
                                   (300, 257, 256, 255)])
def test_gpu_voxel_sums_in_order(ctx, sizes):
    rng = np.random.default_rng(len(sizes) + sizes[0])
    # clusters a unit apart, each within one voxel: the cell is under a tenth
    # and the members lie within a thousandth of a point inside it
    sparse = np.array([[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]] * 50)
    opts = MvsOptions(voxel_rel=0.04)
    owner = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    centre = np.stack([np.arange(len(sizes)) * 1.0 + 0.013, np.full(len(sizes), -2.987), np.full(len(sizes), 5.013)], 1)
    xyz = centre[owner] + rng.uniform(0, 1e-3, (len(owner), 3))
    rgb = rng.integers(0, 256, (len(owner), 3)).astype(np.uint8)
    got_xyz, got_rgb = mvs.fuse_reduce(xyz, rgb, sparse, opts, ctx)
    assert len(got_xyz) == len(sizes)
    for k, n in enumerate(sizes):
        s = np.zeros(3)
        for p in xyz[owner == k]:
            s = s + p
        assert np.array_equal(got_xyz[k], s / n)
        c = rgb[owner == k].astype(np.uint64).sum(0) % 65536
        assert np.array_equal(got_rgb[k], np.minimum(np.floor(c / n + 0.5), 255).astype(np.uint8))

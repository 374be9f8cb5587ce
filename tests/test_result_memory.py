"""Clouds and SIFT frames come back in ordinary arrays: each owns its memory
(none keeps another alive, in-place resize works), in threads too, and a failed
call leaves nothing behind."""
import contextlib
import ctypes as C
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from rustcolmap_b200 import MvsOptions, _abi, mvs, scene, sift
from rustcolmap_b200._lib import RcmvsError


def _ordinary(a):
    assert a.flags.owndata and a.base is None and a.flags.writeable and a.flags.c_contiguous
    first = a[:1].copy()
    a.resize((len(a) + 3,) + a.shape[1:], refcheck=False)
    assert np.array_equal(a[:1], first) and not a[-3:].any()


def test_allocator_hands_out_owned_arrays():
    for field, (dtype, k) in _abi.RESULT_FIELDS.items():
        at = _abi.result_alloc(None, field, 5)
        a = _abi.take_result(field)
        assert a.ctypes.data == at and a.shape == (5, k) and a.dtype == dtype
        a[:] = 7  # unwritten memory may hold NaN
        _ordinary(a)
        assert _abi.take_result(field).shape == (0, k)  # taken once
        assert _abi.result_alloc(None, field, 2**62) is None  # too large: no memory
        assert _abi.take_result(field).shape == (0, k)
    _abi.result_alloc(None, _abi.XYZ, 4)
    _abi.drop_results()
    assert len(_abi.take_result(_abi.XYZ)) == 0


def _image(seed, w=320, h=240):
    return scene.corner_room(seed=seed, n_views=1, w=w, h=h, f=300.0).views[0].rgb


@pytest.mark.gpu
def test_gpu_results_own_their_memory():
    rng = np.random.default_rng(1)
    xyz = rng.uniform(-1, 1, (40000, 3))
    rgb = rng.integers(0, 256, xyz.shape).astype(np.uint8)
    with contextlib.closing(mvs.Context(0)) as ctx:
        f = sift.extract_sift(_image(2), ctx=ctx)
        assert len(f.pts) == len(f.desc) == len(f.colors) > 50
        cloud = mvs.fuse_reduce(xyz, rgb, xyz, MvsOptions(voxel_rel=1e-6), ctx)
        assert len(cloud[0]) == len(cloud[1]) == 40000
        for a in (f.pts, f.desc, f.colors) + cloud:
            _ordinary(a)
        empty = sift.extract_sift(np.zeros((64, 64), np.uint8), ctx=ctx)
        assert empty.pts.shape == (0, 2) and empty.desc.shape == (0, 128) and empty.colors.shape == (0, 3)
        with pytest.raises(RcmvsError):
            mvs.fuse_reduce(xyz, rgb, xyz, MvsOptions(voxel_rel=1e-12), ctx)  # too many cells
        assert len(_abi.take_result(_abi.XYZ)) == 0


@pytest.mark.gpu
def test_gpu_results_in_threads():
    imgs = [_image(k) for k in range(6)]
    ctxs = [mvs.Context(0) for _ in range(3)]
    want = [sift.extract_sift(i, ctx=ctxs[0]) for i in imgs]
    got = sift.extract_sift_many(imgs, ctxs=ctxs)
    for a, b in zip(got, want):
        assert np.array_equal(a.desc, b.desc) and np.array_equal(a.pts, b.pts) and a.desc.flags.owndata
    with ThreadPoolExecutor(3) as ex:
        again = list(ex.map(lambda k: sift.extract_sift(imgs[k], ctx=ctxs[k]), range(3)))
    assert all(np.array_equal(a.colors, b.colors) for a, b in zip(again, want))
    for c in ctxs:
        c.close()


@pytest.mark.gpu
def test_gpu_library_allocates_by_default():
    """Without an allocator the frame's arrays are the library's, released by
    its own call; the same features."""
    img = _image(3)
    with contextlib.closing(mvs.Context(0)) as ctx:
        want = sift.extract_sift(img, ctx=ctx)
        L = ctx._L
        ctx.check(L.rcmvs_ctx_set_result_alloc(ctx.ptr, None, None))
        o, f = sift.SiftOptions().to_c(), _abi.SiftFrame()
        h, w, c = img.shape
        ctx.check(L.rcmvs_extract_sift(ctx.ptr, np.ascontiguousarray(img).ctypes.data, w, h, c, C.byref(o), C.byref(f)))
        d = np.ctypeslib.as_array((C.c_float * (f.n * 128)).from_address(f.desc)).reshape(f.n, 128).copy()
        L.rcmvs_sift_frame_free(C.byref(f))
        assert f.desc is None and np.array_equal(d, want.desc)

"""The stereo kernels' bounded projection (and the staged passes built on it)
against the kernels that run the reference's chain for every window term:
every output bit must agree, over tile edges and remainders, support-view
counts, distorted reference and support cameras, and poses and depth ranges
that leave the projection no bound."""
import numpy as np
import pytest

from rustcolmap_b200 import MvsOptions, mvs, scene
from rustcolmap_b200.types import FLAG_CUDA_GRAPH, FLAG_LOCKSTEP_PASSES, FLAG_NO_REPEAT_SKIP, FLAG_ROW_STEP_INIT

pytestmark = pytest.mark.gpu

CHAIN = FLAG_LOCKSTEP_PASSES | FLAG_ROW_STEP_INIT  # the reference's chain for every term


def _maps(views, jobs, opts, flags):
    ctx = mvs.Context(0)
    ds = mvs.DeviceScene(views, ctx)
    ds.estimate(jobs, MvsOptions(**{**opts.__dict__, "flags": flags}))
    out = [ds.depth(j[0], normals=True) for j in jobs]
    ds.close()
    ctx.close()
    return out


def _same(views, jobs, opts, flags=(0,)):
    want = _maps(views, jobs, opts, CHAIN)
    for f in flags:
        for j, a, b in zip(jobs, _maps(views, jobs, opts, f), want):
            for x, y, name in ((a.depth, b.depth, "depth"), (a.cost, b.cost, "cost"), (a.normal, b.normal, "normal")):
                n = int((x.view(np.uint32) != y.view(np.uint32)).sum())
                assert n == 0, f"flags {f}, view {j[0]} {name}: {n} of {x.size} differ"
    return want


def _scene(w, h, views=5, seed=21, f=None):
    return scene.corner_room(seed=seed, n_views=views, w=w, h=h, f=f or 1.1 * w, arc_deg=40.0, n_patches=60,
                             per_view_sparse=60)


@pytest.mark.parametrize("w,h", [(16, 16), (15, 17), (33, 9), (97, 65), (161, 31), (1, 40)])
@pytest.mark.parametrize("k", [0.0, -0.08])
def test_tile_edges(w, h, k):
    sc = _scene(max(w, 16), max(h, 16))
    for v in sc.views:
        v.cam.k = k
        if w < 16:  # a one-column view: every window cell is clamped
            v.gray, v.rgb, v.w = np.ascontiguousarray(v.gray[:, :w]), np.ascontiguousarray(v.rgb[:, :w]), w
    jobs = [(2, [1, 3, 0], 2.0, 9.0), (0, [1], 2.0, 9.0)]
    _same(sc.views, jobs, MvsOptions(max_dim=4096, num_hyp=16, sweeps=2), (0, FLAG_NO_REPEAT_SKIP, FLAG_CUDA_GRAPH))


@pytest.mark.parametrize("ks", [(0.0, 0.05), (0.05, 0.0), (-0.3, 0.2), (1e-30, 0.0)])
def test_mixed_distortion(ks):
    sc = _scene(120, 88)
    for i, v in enumerate(sc.views):
        v.cam.k = ks[i & 1]
    jobs = [(i, [(i + 1) % 5, (i + 2) % 5, (i + 3) % 5], 1.5, 12.0) for i in range(5)]
    maps = _same(sc.views, jobs, MvsOptions(max_dim=4096, num_hyp=24, sweeps=2))
    assert any((m.depth > 0).any() for m in maps)


@pytest.mark.parametrize("srcs", [1, 2, 9, 32])
def test_source_counts(srcs):
    sc = _scene(72, 50, views=33)
    order = [i for i in range(33) if i != 16]
    order.sort(key=lambda i: abs(i - 16))
    _same(sc.views, [(16, order[:srcs], 2.0, 9.0)], MvsOptions(max_dim=4096, num_hyp=12, sweeps=3))


def test_no_bound():
    """Support views beside, behind and facing the reference view, depths from
    a hundredth of the baseline on, long and short focal lengths, principal
    points far outside the image."""
    sc = _scene(96, 64, views=6)
    v = sc.views
    r180 = np.diag([-1.0, 1.0, -1.0])
    v[1].R, v[1].t = r180 @ v[0].R, r180 @ v[0].t + np.array([0.0, 0.0, 3.0])  # facing
    v[2].t = v[0].R @ (v[0].R.T @ v[0].t) + np.array([0.0, 0.0, -3.0])  # ahead along the axis
    v[2].R = v[0].R
    v[3].cam.cx, v[3].cam.cy = 4000.0, -3000.0
    v[4].cam.f = 9.0
    v[5].cam.f = 30000.0
    jobs = [(0, [1, 2, 3, 4, 5], 0.01, 60.0), (4, [0, 5, 1], 0.05, 40.0), (5, [4, 0], 1.0, 20.0)]
    _same(v, jobs, MvsOptions(max_dim=4096, num_hyp=32, sweeps=3))

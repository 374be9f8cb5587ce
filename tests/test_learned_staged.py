"""The staged learned init (seeds by blocks of 4x4 pixels, the sweep of the
others by packed candidates) against the row-step one, which runs the
reference's chain for every window term: every plane and cost bit, over tile
remainders, quarter-cell remainders, local planes, distortion and both sweep
modes."""
import numpy as np
import pytest

from rustcolmap_b200 import MvsOptions, learned, mvs, scene
from rustcolmap_b200.types import FLAG_INIT_ONLY, FLAG_LOCKSTEP_PASSES, FLAG_SEED_AND_SWEEP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(64, 16), (67, 19), (98, 71), (33, 9), (130, 50)])
@pytest.mark.parametrize("n_local,span,sweep,k,conf", [(1, 0.0, 0, 0.0, 0.3), (3, 0.2, 0, 0.02, 0.3),
                                                       (1, 0.0, FLAG_SEED_AND_SWEEP, -0.05, 0.5),
                                                       (4, 0.8, FLAG_SEED_AND_SWEEP, 0.0, 0.02), (2, 0.1, 0, 0.0, 0.999)])
def test_staged_equals_rows(w, h, n_local, span, sweep, k, conf):
    n = 11
    sc = scene.corner_room(seed=9, n_views=n, w=w, h=h, f=1.2 * w, arc_deg=50.0, n_patches=30, per_view_sparse=80,
                           device=0)
    for v in sc.views:
        v.cam.k = k
    jobs = [(i, [(i + d) % n for d in range(1, m + 1)], 2.0, 9.0) for i, m in enumerate((1, 3, 8, 10))]
    rng = np.random.default_rng(w * 1000 + h + n_local)
    q = (len(jobs), h // 4, w // 4)
    pred = np.zeros(q + (16,), np.float32)
    pred[..., 0] = rng.uniform(-0.5, 1.5, size=q)
    nrm = rng.normal(size=q + (3,))
    nrm[..., 2] = np.abs(nrm[..., 2]) + 0.3
    nrm[rng.uniform(size=q) < 0.15] *= -1
    nrm[rng.uniform(size=q) < 0.05] = 0
    pred[..., 1:4] = nrm
    pred[..., 4] = rng.normal(0.0, 2.0, size=q)
    out = []
    for extra in (0, FLAG_LOCKSTEP_PASSES):
        ctx = mvs.Context(0)
        ds = mvs.DeviceScene(sc.views, ctx)
        opts = MvsOptions(max_dim=4096, num_sources=10, num_hyp=21, cost_thr=2.0,
                          flags=FLAG_INIT_ONLY | sweep | extra)
        seeded = learned.estimate_seeded(ds, jobs, opts, pred, conf_thr=conf, n_local=n_local, span=span)
        out.append((seeded, [ds.depth(j[0], normals=True) for j in jobs]))
        ds.close()
        ctx.close()
    assert out[0][0] == out[1][0]  # 0 where the threshold leaves no seed
    for a, b in zip(out[0][1], out[1][1]):
        for x, y in ((a.depth, b.depth), (a.cost, b.cost), (a.normal, b.normal)):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32))

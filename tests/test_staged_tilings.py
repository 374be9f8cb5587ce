"""The staged passes' tilings, chosen by the size of the batch (16x16 tiles
below 2000, below 18000, above), against the lockstep kernels bit for bit, on
sizes with remainders in both directions."""
import pytest

from rustcolmap_b200 import MvsOptions

from test_bounded_projection import _same, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,jobs", [(249, 121, 1), (249, 257, 7), (257, 249, 8), (641, 603, 11), (641, 603, 12)])
@pytest.mark.parametrize("k", [0.0, 0.03])
def test_batch_sizes(w, h, jobs, k):
    sc = _scene(w, h, views=max(jobs, 4))
    for v in sc.views:
        v.cam.k = k
    n = len(sc.views)
    todo = [(i, [(i + 1) % n, (i + 2) % n], 2.0, 9.0) for i in range(jobs)]
    _same(sc.views, todo, MvsOptions(max_dim=4096, num_hyp=8, sweeps=1))

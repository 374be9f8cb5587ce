"""Training labels are floats in the caller's buffer: any float-aligned address
gives the step that a 16-byte aligned one gives."""
import contextlib

import numpy as np
import pytest

from rustcolmap_b200 import learned, mvs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 17, 9)])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_labels_at_float_alignment(shape, shift):
    """One pixel: every sum has one term, so equal bits.  More: the same terms in
    another order (atomic adds), at most 306 * 2^-24 = 2e-5 of their absolute
    sum; 1e-3 of the norm leaves room for cancellation."""
    import torch
    n, h, w = shape
    rng = np.random.default_rng(shift)
    x = rng.random((n, h, w, learned.COSTVOL_C), dtype=np.float32)
    x[..., 33:] = 0
    lab = np.zeros((n, h, w, learned.LABEL_C), np.float32)
    lab[..., 0] = rng.random((n, h, w))
    lab[..., 1:4] = rng.random((n, h, w, 3)) + 0.1
    lab[..., 4] = 1
    lab[..., 5] = 0.05
    xd = torch.from_numpy(x).to(torch.bfloat16).cuda()
    buf = torch.zeros(lab.size + 8, dtype=torch.float32, device="cuda")
    assert buf.data_ptr() % 16 == 0
    got = []
    with contextlib.closing(mvs.Context(0)) as ctx, contextlib.closing(learned.ProposalNet(ctx, seed=5)) as net:
        for at in (0, shift):
            buf[at:at + lab.size] = torch.from_numpy(lab.reshape(-1)).cuda()
            torch.cuda.synchronize()
            got.append(net.train_step(xd.data_ptr(), buf.data_ptr() + 4 * at, n, h, w, 0.0, apply=False, grads=True))
    (l0, g0), (l1, g1) = got
    if n * h * w == 1:
        assert l0 == l1 and np.array_equal(g0, g1)
    assert abs(l0 - l1) <= 1e-3 * abs(l0) and np.linalg.norm(g0 - g1) <= 1e-3 * np.linalg.norm(g0)

"""Weight, bias and data gradients of the network's tensor-core kernels at
sizes around their 16 x 8 tiles, against the FP32 oracle."""
import numpy as np
import pytest

from oracle import net_oracle
from rustcolmap_b200 import learned, mvs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (1, 16, 8), (2, 17, 9), (1, 15, 40), (3, 5, 23), (1, 33, 70)])
def test_gradients_at_tile_edges(n, h, w):
    """The oracle rounds to BF16 where the kernels do, so what is left is the
    order of FP32 sums and the few roundings it moves: the bounds are
    test_learned's for a whole step (gradient cosine and relative error per
    layer)."""
    import torch
    rng = np.random.default_rng(100 * h + w)
    x = np.zeros((n, h, w, learned.COSTVOL_C), np.float32)
    x[..., :33] = rng.random((n, h, w, 33), dtype=np.float32)
    lab = np.zeros((n, h, w, learned.LABEL_C), np.float32)
    lab[..., 0] = rng.random((n, h, w))
    nrm = rng.standard_normal((n, h, w, 3)) + [0, 0, 2]
    lab[..., 1:4] = nrm / np.linalg.norm(nrm, axis=-1, keepdims=True)
    lab[..., 4] = 1
    lab[..., 5] = 0.05
    ctx = mvs.Context(0)
    net = learned.ProposalNet(ctx, seed=3)
    p = net.params()
    xd = torch.from_numpy(x).cuda().to(torch.bfloat16).contiguous()
    ld = torch.from_numpy(lab).cuda()
    torch.cuda.synchronize()
    loss, g = net.train_step(xd.data_ptr(), ld.data_ptr(), n, h, w, 1e-3, apply=False, grads=True)
    want_loss, want = net_oracle.gradients(p, x, lab)
    assert abs(loss - want_loss) <= 0.01 * abs(want_loss)
    lay, _ = net_oracle.param_layout()
    for (wo, wn), (bo, bn), _, _ in lay:
        for o, k in ((wo, wn), (bo, bn)):
            a, b = g[o:o + k].astype(np.float64), want[o:o + k].astype(np.float64)
            if np.linalg.norm(b) < 1e-6:
                assert np.linalg.norm(a) < 1e-4
                continue
            cos = a @ b / (np.linalg.norm(a) * np.linalg.norm(b))
            rel = np.linalg.norm(a - b) / np.linalg.norm(b)
            assert cos > 0.995 and rel < 0.06, f"offset {o}: cosine {cos:.5f}, relative error {rel:.4f}"
    net.close()
    ctx.close()

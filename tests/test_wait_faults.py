"""A bounded tensor-core wait that ran out (the diagnostic waits on a barrier
nothing arrives on, which sets the context's fault word as the kernels do):
a call whose results depend on such waits returns an error in their place."""
import contextlib

import numpy as np
import pytest

from oracle import oracle
from rustcolmap_b200 import learned, mvs, sift
from rustcolmap_b200._lib import RcmvsError

pytestmark = pytest.mark.gpu


def _batch(seed):
    import torch
    rng = np.random.default_rng(seed)
    n, h, w = 1, 20, 19
    x = rng.random((n, h, w, learned.COSTVOL_C), dtype=np.float32)
    x[..., 33:] = 0
    lab = np.zeros((n, h, w, learned.LABEL_C), np.float32)
    lab[..., 0] = rng.random((n, h, w))
    lab[..., 3:5] = 1
    lab[..., 5] = 0.05
    return torch.from_numpy(x).to(torch.bfloat16).cuda(), torch.from_numpy(lab).cuda(), (n, h, w)


def test_train_step_takes_no_step():
    xd, ld, shape = _batch(4)
    with contextlib.closing(mvs.Context(0)) as ctx, contextlib.closing(mvs.Context(0)) as other, \
            contextlib.closing(learned.ProposalNet(ctx, seed=9)) as net:
        p = net.params()
        ctx.diag_wait_timeout(1_000_000)
        with pytest.raises(RcmvsError, match="timed out"):
            net.train_step(xd.data_ptr(), ld.data_ptr(), *shape, 1e-2, grads=True)
        other.synchronize()  # another context's word is not touched
        assert np.array_equal(net.params(), p)
        ctx.synchronize()  # reported once
        net.train_step(xd.data_ptr(), ld.data_ptr(), *shape, 1e-2)
        moved = np.abs(net.params() - p).max()
        assert 0 < moved <= 1.01e-2  # one first Adam step


def test_matching_reads_no_unwritten_entry():
    """The search's entries are kept in a buffer that earlier calls leave
    larger indices in; with the fault set, no kernel follows them."""
    def descs(n, seed):
        d = np.random.default_rng(seed).random((n, 128), dtype=np.float32)
        return np.ascontiguousarray(d / np.linalg.norm(d, axis=1, keepdims=True))

    a, b = descs(2100, 1), descs(2050, 2)
    b[:400] = a[1700:2100]
    with contextlib.closing(mvs.Context(0)) as ctx:
        sift.match_pairs([a, descs(9000, 3)], [(0, 1), (1, 0)], 1.0, ctx)
        ctx.diag_wait_timeout(1_000_000)
        with pytest.raises(RcmvsError, match="timed out"):
            sift.match_pairs([a, b], [(0, 1)], 0.8, ctx)
        ctx.synchronize()  # reported once
        (ga, gb), = sift.match_pairs([a, b], [(0, 1)], 0.8, ctx)
        oa, ob = oracle.match_pair(a, b, 0.8)
        assert len(oa) >= 400 and np.array_equal(ga, oa) and np.array_equal(gb, ob)

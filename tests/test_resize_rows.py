"""The vertical resize pass at the edges of its rows of 512 elements, four to
a thread, for every channel count and row remainder, against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle
from rustcolmap_b200 import mvs


@pytest.mark.gpu
@pytest.mark.parametrize("channels", [1, 2, 3, 4])
@pytest.mark.parametrize("w", [1, 3, 4, 127, 128, 170, 171, 172, 512, 513, 516, 1025])
def test_gpu_row_edges(channels, w):
    img = np.random.default_rng(w * 8 + channels).integers(0, 256, (37, w, channels), dtype=np.uint8)
    ctx = mvs.Context(0)
    for mw, mh in ((max(w // 2, 1), 17), (w + 5, 80), (w, 1)):
        gray, rgb = mvs.resize_view(img, mw, mh, ctx)
        og, orgb = oracle.resize_view(img, mw, mh)
        assert np.array_equal(gray, og) and np.array_equal(rgb, orgb)
    ctx.close()

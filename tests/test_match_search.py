"""The tensor-core descriptor search against the CPU oracle: block edges and
remainders, target counts around its four candidates, scales outside the
packed range (the FP32 kernels), and near-equal distances past the candidate
list (rescans, then the FP32 kernels)."""
import numpy as np
import pytest

from oracle import oracle
from rustcolmap_b200 import mvs, sift

pytestmark = pytest.mark.gpu


def _descs(n, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    d = rng.random((n, 128), dtype=np.float32) ** 3
    d = np.minimum(d / np.linalg.norm(d, axis=1, keepdims=True), 0.2)
    return np.ascontiguousarray(d / np.linalg.norm(d, axis=1, keepdims=True) * np.float32(scale))


def _check(sets, ratio):
    """Every ordered pair of the sets, in one call with a pair of large frames
    that takes it past the tensor-core search's smallest size, and alone."""
    small = [(i, j) for i in range(len(sets)) for j in range(len(sets)) if i != j]
    big = sets + [_descs(2100, 90), _descs(2050, 91)]
    m = len(sets)
    n = _compare(big, small + [(m, m + 1), (m, 0), (0, m + 1)], ratio)
    assert _compare(sets, small, ratio) <= n
    return n


def _compare(sets, pairs, ratio):
    ctx = mvs.Context(0)
    got = sift.match_pairs(sets, pairs, ratio, ctx)
    n = 0
    for (i, j), (ga, gb) in zip(pairs, got):
        oa, ob = oracle.match_pair(sets[i], sets[j], ratio)
        assert np.array_equal(ga, oa) and np.array_equal(gb, ob), f"pair {i}, {j}: {len(ga)} / {len(oa)} matches"
        n += len(ga)
    ctx.close()
    return n


def _related(counts, seed, scale=1.0, noise=0.1):
    rng = np.random.default_rng(seed)
    base = _descs(max(counts) + 8, seed)
    out = []
    for k, n in enumerate(counts):
        d = _descs(n, seed + 1 + k)
        m = n // 2
        d[:m] = base[rng.permutation(len(base))[:m]] * (1 + noise * (rng.random((m, 128)) - 0.5))
        out.append(np.ascontiguousarray(d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-9) * scale,
                                        dtype=np.float32))
    return out


@pytest.mark.parametrize("counts", [(1, 2, 3), (4, 5, 0, 6), (127, 128, 129), (255, 257, 384, 1), (1000, 700)])
@pytest.mark.parametrize("ratio", [0.8, 1.0])
def test_block_edges(counts, ratio):
    n = _check(_related(counts, 7), ratio)
    assert n > 0 or max(counts) < 8


@pytest.mark.parametrize("scale", [1e-20, 1e-4, 0.05, 0.5, 3000.0])
def test_scales(scale):
    sets = _related((200, 150, 129), 11)
    _check([np.ascontiguousarray(s * np.float32(scale)) for s in sets], 0.9)


def test_mixed_range_frames():
    sets = _related((140, 90, 60), 13)
    sets[1] = sets[1].copy()
    sets[1][5] *= np.float32(1e6)
    sets[2] = sets[2].copy()
    sets[2][3, 7] = np.inf
    _check(sets, 0.8)


@pytest.mark.parametrize("copies,n", [(3, 64), (6, 64), (6, 600)])
def test_equal_descriptors(copies, n):
    """Every descriptor `copies` times: with six the four candidates cannot
    hold the ties (few such queries: rescans; many: the FP32 kernels)."""
    base = _descs(n, 17)
    a = np.ascontiguousarray(np.repeat(base, copies, axis=0))
    b = np.ascontiguousarray(np.concatenate([base, _descs(40, 18)]))
    for ratio in (0.8, 1.0, 1.2):
        _check([a, b], ratio)
    near = np.ascontiguousarray(a * (1 + 1e-6 * np.random.default_rng(1).random(a.shape)), dtype=np.float32)
    _check([near, b], 1.0)

"""The tensor-core search's approximate distances against 64-bit ones: within
the derived 52 u S^2 + 2^-26 S (u = 2^-24, S = |q| + |t|) and so within the
bound the decisions use, on descriptors made to lose much in the accumulation
(one large product and many that its exponent cuts off), near duplicates,
components at the packed range's end and over many magnitudes; and decisions
whose nearest two targets share a column pair."""
import contextlib

import numpy as np
import pytest

from oracle import oracle
from rustcolmap_b200 import mvs, sift

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with contextlib.closing(mvs.Context(0)) as c:
        yield c


def _check(ctx, q, targets):
    q = np.ascontiguousarray(q, np.float32)
    worst = 0.0
    for t in np.ascontiguousarray(targets, np.float32):
        t = t[None]
        approx, bound = np.empty(len(q), np.float32), np.empty(len(q), np.float32)
        ctx.check(ctx._L.rcmvs_diag_match_distances(ctx.ptr, q.ctypes.data, len(q), t.ctypes.data, 1,
                                                    approx.ctypes.data, bound.ctypes.data))
        q64, t64 = q.astype(np.float64), t.astype(np.float64)
        err = np.abs(approx - ((q64 - t64) ** 2).sum(1))
        s = np.sqrt((q64 ** 2).sum(1)) + np.sqrt((t64 ** 2).sum())
        limit = 52 * 2.0 ** -24 * s ** 2 + 2.0 ** -26 * s
        assert (err <= limit).all(), f"{(err / limit).max():.3f} of the derived error"
        assert (limit <= bound).all()
        worst = max(worst, float((err / limit).max()))
    return worst


def _one_large(rng, n, r, pos, sign, jitter):
    x = np.full((n, 128), 2.0 ** (-r / 2)) * (1 - jitter * rng.random((n, 128)))
    x[:, pos] = 1 + 0.02 * rng.random(n)
    x *= np.where(np.arange(128) == pos, 1.0, sign)
    return x


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("pos", [0, 15, 16, 100])
def test_one_large_product(ctx, pos, sign):
    rng = np.random.default_rng(pos)
    for r in range(12, 30):
        for jitter in (0.0, 0.02, 0.5):
            q = _one_large(rng, 200, r, pos, 1.0, jitter) * rng.uniform(0.7, 1.0, (200, 1))
            _check(ctx, q, _one_large(rng, 4, r, pos, sign, jitter) * rng.uniform(0.7, 1.0, (4, 1)))


@pytest.mark.parametrize("scale", [1e-4, 1.0, 30.0, 999.0])
def test_magnitudes(ctx, scale):
    rng = np.random.default_rng(3)
    worst = 0.0
    for kind in range(6):
        e = [np.zeros(128), rng.uniform(-14, 0, 128), np.repeat(rng.uniform(-14, 0, 8), 16),
             np.sort(rng.uniform(-14, 0, 128))[::-1], np.sort(rng.uniform(-14, 0, 128)),
             np.where(np.arange(128) < 3, 0, -10.0)][kind]
        for sg in (np.ones(128), rng.choice([-1.0, 1.0], 128)):
            q = scale * 2.0 ** e * rng.uniform(0.7, 1.0, (300, 128))
            t = scale * sg * 2.0 ** e * rng.uniform(0.7, 1.0, (6, 128))
            worst = max(worst, _check(ctx, q, t), _check(ctx, q, q[:6] * (1 + 1e-4 * rng.standard_normal((6, 128)))))
    assert worst > 0.01  # the cases are not trivial


@pytest.mark.parametrize("n", [256, 255])
@pytest.mark.parametrize("ratio", [0.8, 1.0, 1.1])
def test_nearest_two_share_a_column_pair(ctx, n, ratio):
    """Targets 2i and 2i + 1 near query i, one of them nearer, or equal."""
    rng = np.random.default_rng(n)

    def unit(m):
        d = rng.random((m, 128)) ** 3
        return d / np.linalg.norm(d, axis=1, keepdims=True)

    base, off = unit(2200), unit(2200)
    b = np.repeat(base[: (n + 1) // 2], 2, axis=0)[:n]
    gap = np.where(np.arange(n) % 2, 0.05, np.array([0.02, 0.05, 0.05 * (1 + 1e-6), 0.2])[np.arange(n) // 2 % 4])
    b = b + gap[:, None] * np.repeat(off[: (n + 1) // 2], 2, axis=0)[:n]
    sets = [np.ascontiguousarray(base, np.float32), np.ascontiguousarray(np.concatenate([b, unit(2100)]), np.float32)]
    (ga, gb), (ha, hb) = sift.match_pairs(sets, [(0, 1), (1, 0)], ratio, ctx)
    for g, (i, j) in (((ga, gb), (0, 1)), ((ha, hb), (1, 0))):
        oa, ob = oracle.match_pair(sets[i], sets[j], ratio)
        assert np.array_equal(g[0], oa) and np.array_equal(g[1], ob)
    assert len(ga) >= n // 8

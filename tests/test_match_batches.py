"""A large batch of pairs: frames uploaded in groups while earlier pairs are
searched, and matches packed on the device from 16384 rows on, in the pairs'
own order (reversed, repeated and self pairs, frames without descriptors)."""
import numpy as np
import pytest

from test_match_search import _compare, _descs, _related

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [16383, 16384, 16800])
def test_packed_matches(rows):
    sets = _related((2048, 0, 1030, 257, 2048, 700), 31)
    sets.append(np.ascontiguousarray(sets[4][::-1]))
    pairs = [(4, 6), (0, 4), (1, 0), (2, 1), (5, 3), (0, 4), (3, 3), (6, 0), (2, 5), (4, 2)]
    used = sum(len(sets[a]) for a, _ in pairs)
    assert used < rows
    sets.append(_descs(rows - used, 32))  # the last pair makes up the rows
    assert _compare(sets, pairs + [(7, 5)], 0.9) > 2048


def test_packed_matches_fp32():
    """Ties past the candidate lists: the FP32 kernels' answers, packed."""
    a = np.ascontiguousarray(np.repeat(_descs(400, 3), 6, axis=0))
    sets = [a, np.ascontiguousarray(a[::-1]), _descs(2100, 5)]
    _compare(sets, [(0, 1), (1, 2), (2, 0), (0, 2), (1, 0), (0, 0), (1, 1)], 1.0)

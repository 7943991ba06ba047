"""The comparison's label pairs counted by community (one warp, one block, or
sorted, by the community's size) against the oracle: integers, exact."""
import numpy as np
import pytest

from grappolo_b200 import louvain
from _golden import COMPARE_FLOATS, COMPARE_INTS

pytestmark = pytest.mark.gpu


def _sizes(sizes, pad=0):
    """Labels of communities of these sizes, and singletons after them."""
    a = np.repeat(np.arange(len(sizes)), sizes)
    return np.concatenate([a, len(sizes) + np.arange(pad)])


@pytest.mark.parametrize('sizes,pad', [
    ([1], 0), ([2], 0), ([1, 1, 1], 0), ([31, 32, 33], 0),      # single warps and rounds
    ([383, 384, 385], 0),                                       # warp table to block table
    ([6143, 6144], 0), ([6143, 6144, 6145], 0),                 # block table to sorting
    ([6145, 20000, 8192, 8193], 3000),                          # several sorted, many chunks
    ([40000], 4000),                                            # nearly all in one
    ([30000], 0),                                               # by keys: one community
])
@pytest.mark.parametrize('noise', [0.0, 0.3, 1.0])
@pytest.mark.parametrize('swap', [False, True])
def test_group_sizes(oracle, sizes, pad, noise, swap):
    rng = np.random.default_rng(len(sizes) + pad)
    a = _sizes(sizes, pad)
    a = a[rng.permutation(len(a))]
    b = a.copy()
    flip = rng.random(len(a)) < noise
    b[flip] = rng.integers(0, a.max() + 1, int(flip.sum()))  # no more communities than a has
    C1, C2 = (b, a) if swap else (a, b)
    st, x, y = louvain.computeCommunityComparisons(C1, C2)
    o, ox, oy = oracle.compare(C1, C2)
    for k in COMPARE_INTS:
        assert st[k] == o[k], k
    for k in COMPARE_FLOATS:
        assert st[k] == o[k] or (np.isnan(st[k]) and np.isnan(o[k])), k
    assert np.array_equal(x, ox) and np.array_equal(y, oy)


@pytest.mark.parametrize('n', [1, 31, 33, 5000])
def test_labels_with_gaps_and_minus_one(oracle, n):
    """Ids with large gaps (more ids than vertices: counted by sorted keys),
    and -1 entries on both sides."""
    rng = np.random.default_rng(n)
    for top in (3, n // 20 + 2, 10 * n + 7):
        C1, C2 = rng.integers(0, top, n), rng.integers(0, top, n)
        C1[rng.random(n) < 0.1] = -1
        C2[rng.random(n) < 0.1] = -1
        C1[0] = C2[0] = 1
        st, x, y = louvain.computeCommunityComparisons(C1, C2)
        o, ox, oy = oracle.compare(C1, C2)
        for k in COMPARE_INTS:
            assert st[k] == o[k], k
        assert np.array_equal(x, ox) and np.array_equal(y, oy)

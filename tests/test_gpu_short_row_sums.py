"""Fast mode on real weights: the candidates of a short row are weighed against one
own-community sum, whichever lane adds it, and it is the sum in entry order.

Eight vertices make a group; v's row is (u1, a1, a2, u2, u3, b1, b2), weights
x1, 0.28, 0.28, x2, x3, 0.28, 0.28.  v joins u1 first (the heaviest single
vertex), u2 and u3 follow it, and {a1, a2} and {b1, b2} close up.  In the second
sweep both pairs offer v the same gain to the last bit, so v takes the smaller
community id, the a pair's.  A lane that adds x2 + x3 + x1 instead of
x1 + x2 + x3 sees another gain, and the tie is lost.
"""
import numpy as np
import pytest

from grappolo_b200 import graphs, louvain

pytestmark = pytest.mark.gpu

U1, A1, A2, U2, U3, B1, B2, V = range(8)


def _groups(n, seed):
    rng = np.random.default_rng(seed)
    x1 = rng.uniform(0.29, 0.4, n)
    x2, x3 = rng.uniform(0.001, 0.07, n), rng.uniform(0.001, 0.07, n)
    side = np.full(n, 0.28)
    tie = np.full(n, 5.0)
    rows = [(V, U1, x1), (V, A1, side), (V, A2, side), (V, U2, x2), (V, U3, x3), (V, B1, side),
            (V, B2, side), (A1, A2, tie), (B1, B2, tie)]
    base = 8 * np.arange(n)
    u = np.concatenate([base + a for a, _, _ in rows])
    v = np.concatenate([base + b for _, b, _ in rows])
    g = graphs.csr_from_undirected(8 * n, u, v, np.concatenate([w for _, _, w in rows]))
    entry, other = (x1 + x2) + x3, (x2 + x3) + x1
    assert (entry != other).mean() > 0.1  # the order shows
    color = np.tile([1, 2, 1, 1, 1, 2, 1, 0], n)  # v, then the u and one of each pair, the rest
    return g, color


@pytest.mark.parametrize('n', [40, 3000])
@pytest.mark.parametrize('threads', [1, 16])  # the ordered sweeps, and fast mode's
def test_ties_stay_ties(n, threads):
    g, color = _groups(n, seed=n)
    _, C, _, _ = louvain.algoLouvainWithDistOneColoring(g, color, 3, thresh=1e-6,
                                                        nThreads=threads)
    C = C.reshape(n, 8)
    assert np.array_equal(C[:, A1], C[:, A2]) and np.array_equal(C[:, B1], C[:, B2])
    assert np.array_equal(C[:, V], C[:, A1])

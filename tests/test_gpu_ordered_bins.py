"""Verify mode on real-valued weights: steps whose rows of one length are just few
enough for the launch all bins share, and one more (a launch of their own), beside
a long row in the shared one.  Bit for bit against the oracle."""
import numpy as np
import pytest

from grappolo_b200 import graphs, louvain

pytestmark = pytest.mark.gpu

WARPS = 2 * 8 * 148  # of the shared launch; a bin with over 2 items for each goes alone


def _ring(n, degree, seed, hub):
    """n vertices of `degree` ring neighbours under shuffled ids and, with hub, one more vertex
    joined to 600 of them that then have one entry more."""
    rng = np.random.default_rng(seed)
    ids = rng.permutation(n)
    i = np.repeat(np.arange(n), degree // 2)
    j = (i + np.tile(np.arange(1, degree // 2 + 1), n)) % n
    u, v = ids[i], ids[j]
    if hub:
        u = np.concatenate([u, np.full(600, n)])
        v = np.concatenate([v, rng.choice(n, 600, replace=False)])
    return graphs.csr_from_undirected(n + hub, u, v, 1.0 - rng.random(u.size))


@pytest.mark.parametrize('degree,per_item', [(4, 8), (8, 4), (16, 2), (32, 1), (40, 1)])
@pytest.mark.parametrize('more', [0, 1])
@pytest.mark.parametrize('hub', [0, 1])
def test_one_step(degree, per_item, more, hub, oracle):
    g = _ring(2 * WARPS * per_item + more, degree, seed=degree, hub=hub)
    C, st = louvain.runMultiPhaseBasic(g, numThreads=1, stats=True)
    Co, so, _ = oracle.run_multiphase_basic(g)
    assert np.array_equal(C, Co)
    assert st['final_modularity'] == pytest.approx(so['final_mod'], rel=1e-9)


@pytest.mark.parametrize('nv', [9000, 60000])
def test_colour_classes(nv, oracle):
    """Large classes of short rows: several own launches a class."""
    g = _ring(nv, 20, seed=nv, hub=1)
    C, st = louvain.runMultiPhaseColoring(g, numThreads=1, stats=True)
    Co, so, _ = oracle.run_multiphase_coloring(g)
    assert np.array_equal(C, Co)
    assert st['final_modularity'] == pytest.approx(so['final_mod'], rel=1e-9)

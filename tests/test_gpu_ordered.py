"""Verify mode on real-valued weights (ordered sums) at the kernels' edges, bit
for bit against the oracle: rows across the staging chunk and the worker
limits, repeated self-loops inside a row, and colour classes on both sides of
the size that one block totals by itself.
"""
import numpy as np
import pytest

from grappolo_b200 import graphs, louvain

pytestmark = pytest.mark.gpu


def _graph(nv, hub_degs, seed, loops, mean=3.0):
    rng = np.random.default_rng(seed)
    n = int(mean * nv / 2)
    u, v = [rng.integers(0, nv, n)], [rng.integers(0, nv, n)]
    for k, d in enumerate(hub_degs):
        u.append(np.full(d, k))
        v.append(rng.choice(np.arange(50, nv), d, replace=False))
    u, v = np.concatenate(u), np.concatenate(v)
    g = graphs.csr_from_undirected(nv, u, v, 1.0 - rng.random(u.size))
    if not loops:
        return g
    # the first hubs get several self-loop entries, at random places of their unsorted rows
    h, t, w = g.heads(), g.tail, g.weight
    ids = np.repeat(np.arange(len(hub_degs)), loops)
    h, t = np.concatenate([h, ids]), np.concatenate([t, ids])
    w = np.concatenate([w, 1.0 - rng.random(ids.size)])
    o = np.lexsort((rng.random(h.size), h))
    ptr = np.zeros(nv + 1, dtype=np.int64)
    np.cumsum(np.bincount(h, minlength=nv), out=ptr[1:])
    return graphs.CSRGraph(ptr, t[o], w[o])


def _check(g, oracle, coloring):
    run = louvain.runMultiPhaseColoring if coloring else louvain.runMultiPhaseBasic
    ref = oracle.run_multiphase_coloring if coloring else oracle.run_multiphase_basic
    C, st = run(g, numThreads=1, stats=True)
    Co, so, _ = ref(g)
    assert np.array_equal(C, Co)
    assert st['final_modularity'] == pytest.approx(so['final_mod'], rel=1e-9)


@pytest.mark.parametrize('coloring', [True, False])
@pytest.mark.parametrize('loops', [0, 3])
@pytest.mark.parametrize('deg', [127, 128, 511, 512, 513, 1023, 1025, 4090, 4097, 6000])
def test_row_lengths(deg, loops, coloring, oracle):
    _check(_graph(8000, [deg, deg], seed=deg, loops=loops), oracle, coloring)


@pytest.mark.parametrize('nv', [700, 4096, 6000, 20000])
def test_class_sizes(nv, oracle):
    """Sparse graphs: the first colour classes hold most vertices."""
    _check(_graph(nv, [], seed=nv, loops=0), oracle, True)

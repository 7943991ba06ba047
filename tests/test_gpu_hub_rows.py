"""Long rows of the sweep (whole-warp, team, block rows; hub chunks and
partitions) at their edges, against the oracle.

Weights are integers, so every sum is exact in any order and verify mode must
equal the oracle bit for bit: communities, modularity, iteration counts.
"""
import numpy as np
import pytest

from grappolo_b200 import _lib, graphs, louvain

pytestmark = pytest.mark.gpu


def _mix32(x):
    x = x.astype(np.uint64)
    m = np.uint64(0xffffffff)
    x ^= x >> np.uint64(16); x = (x * np.uint64(0x7feb352d)) & m
    x ^= x >> np.uint64(15); x = (x * np.uint64(0x846ca68b)) & m
    x ^= x >> np.uint64(16)
    return x


def _with_hubs(nv, rows, seed, loops=True):
    """Sparse random edges plus one row of exactly about each given length."""
    rng = np.random.default_rng(seed)
    u = [rng.integers(0, nv, 2 * nv)]
    v = [rng.integers(0, nv, 2 * nv)]
    for hub, neigh in rows:
        u.append(np.full(len(neigh), hub))
        v.append(np.asarray(neigh))
    u, v = np.concatenate(u), np.concatenate(v)
    g = graphs.csr_from_undirected(nv, u, v, rng.integers(1, 9, u.size).astype(np.float64))
    if not loops:
        return g
    # self-loops on the hubs (they count in Counter[own] and in the self-loop sum)
    h, t, w = g.heads(), g.tail, g.weight
    ids = np.array([r[0] for r in rows])
    h, t = np.concatenate([h, ids]), np.concatenate([t, ids])
    w = np.concatenate([w, np.full(ids.size, 3.0)])
    o = np.lexsort((t, h))
    ptr = np.zeros(nv + 1, dtype=np.int64)
    np.cumsum(np.bincount(h, minlength=nv), out=ptr[1:])
    return graphs.CSRGraph(ptr, t[o], w[o])


def _check(g, oracle, coloring=True):
    run = louvain.runMultiPhaseColoring if coloring else louvain.runMultiPhaseBasic
    C, st = run(g, numThreads=1, stats=True)
    Co, so, _ = (oracle.run_multiphase_coloring if coloring else oracle.run_multiphase_basic)(g)
    assert np.array_equal(C, Co)
    assert st['final_modularity'] == pytest.approx(so['final_mod'], rel=1e-12)


@pytest.mark.parametrize('coloring', [True, False])
@pytest.mark.parametrize('deg', [30, 33, 120, 127, 128, 255, 256, 511, 512, 513, 1023, 1024, 4090,
                                 4095, 4096, 4097, 5000, 9000])
def test_row_lengths(deg, coloring, oracle):
    """Two rows whose length crosses each worker's limits (the random edges add a few entries)."""
    nv = 12000
    rng = np.random.default_rng(deg)
    rows = [(7, rng.choice(np.arange(100, nv), deg, replace=False)),
            (11, rng.choice(np.arange(100, nv), deg, replace=False))]
    _check(_with_hubs(nv, rows, seed=deg), oracle, coloring)


@pytest.mark.parametrize('block_max', ['127', '1000'])
def test_many_small_hubs(block_max, oracle, monkeypatch):
    """Every row above the forced limit is a hub: many hubs, one to a few chunks each."""
    monkeypatch.setenv('GRAPPOLO_B200_BLOCK_MAX', block_max)
    nv = 6000
    rng = np.random.default_rng(5)
    rows = [(k, rng.choice(np.arange(100, nv), 130 + 97 * k, replace=False)) for k in range(40)]
    _check(_with_hubs(nv, rows, seed=6), oracle)


@pytest.mark.parametrize('deg', [6000, 16384, 40000])
def test_one_partition_gets_every_community(deg, oracle):
    """All of a hub's neighbours fall in one partition: more distinct communities than a merge
    holds at once, so it splits them into shares."""
    nv = 400000
    ids = np.arange(100, nv)
    ids = ids[(_mix32(ids) & np.uint64(31)) == 0]
    neigh = np.random.default_rng(deg).choice(ids, min(deg, ids.size), replace=False)
    _check(_with_hubs(nv, [(3, neigh)], seed=deg), oracle)


def test_launch_per_kernel_path(oracle, monkeypatch):
    """The same hubs without the persistent kernel."""
    monkeypatch.setenv('GRAPPOLO_B200_PERSISTENT', '0')
    nv = 30000
    rng = np.random.default_rng(9)
    rows = [(k, rng.choice(np.arange(100, nv), d, replace=False))
            for k, d in enumerate([4100, 5000, 8191, 8192, 20000])]
    _check(_with_hubs(nv, rows, seed=9), oracle)


def test_lower_grouping_is_the_hub_limit_not_the_workers(monkeypatch):
    """Fast mode's merged classes depend on the grouping limit alone: a tuned run equals one
    whose workers use the other limit."""
    monkeypatch.setenv('GRAPPOLO_B200_COLORING', 'id')
    monkeypatch.setenv('GRAPPOLO_B200_AUTOTUNE_MIN', '0')
    g = graphs.rmat(15, seed=3)
    g = graphs.CSRGraph(g.ptr, g.tail, np.ceil(g.weight * 16))
    runs = [louvain.run_multiphase_csr(g, mode=_lib.GLV_MODE_FAST) for _ in range(2)]
    assert np.array_equal(runs[0][0], runs[1][0])
    assert runs[0][1]['final_modularity'] == runs[1][1]['final_modularity']

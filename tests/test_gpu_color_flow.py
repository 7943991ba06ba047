"""The dataflow colouring against sequential first-fit in priority order.

Colours are whole numbers fixed by the priorities, so every comparison is
exact.  The graphs sit at the edges of the kernel: colours across the 32-colour
word and its bitmap words, rows across the task size, chains longer than a
warp keeps to itself, repeated entries, self-loops and unsorted rows.
"""
import numpy as np
import pytest

from grappolo_b200 import _lib, graphs, louvain

pytestmark = pytest.mark.gpu

SEED = 0x5bd1e995


def _mix32(x):
    x = x.astype(np.uint64)
    m = np.uint64(0xffffffff)
    x ^= x >> np.uint64(16); x = (x * np.uint64(0x7feb352d)) & m
    x ^= x >> np.uint64(15); x = (x * np.uint64(0x846ca68b)) & m
    x ^= x >> np.uint64(16)
    return x


def _first_fit(g, hashed):
    ids = np.arange(g.num_vertices, dtype=np.int64)
    order = np.lexsort((ids, _mix32(ids ^ SEED))) if hashed else ids
    col = np.full(g.num_vertices, -1, dtype=np.int32)
    for v in order:
        t = g.tail[g.ptr[v]:g.ptr[v + 1]]
        used = col[t[t != v]]
        used = np.unique(used[used >= 0])
        gap = np.nonzero(used != np.arange(used.size))[0]
        col[v] = gap[0] if gap.size else used.size
    return col


def _edges(nv, u, v):
    return graphs.csr_from_undirected(nv, np.asarray(u), np.asarray(v))


def _clique(n, extra=3):
    u, v = np.triu_indices(n, k=1)
    return _edges(n + extra, u, v)


def _star(n):  # the hub in the middle of the ids: lower and higher neighbours
    leaf = np.delete(np.arange(n), n // 2)
    return _edges(n, np.full(n - 1, n // 2), leaf)


def _path(n):
    return _edges(n, np.arange(n - 1), np.arange(1, n))


def _core(n, hubs, seed):
    """A dense core of `hubs` low ids joined to many others (rows of several tasks)."""
    rng = np.random.default_rng(seed)
    u, v = np.triu_indices(hubs, k=1)
    keep = rng.random(u.size) < 0.8
    a = rng.integers(0, hubs, 40 * n // 10)
    b = rng.integers(hubs, n, 40 * n // 10)
    return _edges(n, np.concatenate([u[keep], a]), np.concatenate([v[keep], b]))


def _messy(seed):
    """Unsorted rows with repeated entries (in both directions) and self-loops."""
    g = graphs.rmat(9, edge_factor=6, seed=seed)
    rng = np.random.default_rng(seed)
    h = g.heads()
    pick = rng.integers(0, g.nnz, g.nnz // 3)
    loop = rng.integers(0, g.num_vertices, 50)
    src = np.concatenate([h, h[pick], g.tail[pick], loop])
    dst = np.concatenate([g.tail, g.tail[pick], h[pick], loop])
    order = np.lexsort((rng.random(src.size), src))
    ptr = np.zeros(g.num_vertices + 1, dtype=np.int64)
    np.cumsum(np.bincount(src, minlength=g.num_vertices), out=ptr[1:])
    return graphs.CSRGraph(ptr, dst[order], np.ones(src.size))


CASES = {
    'one': lambda: graphs.CSRGraph(np.zeros(2, np.int64), np.zeros(0, np.int64), np.zeros(0)),
    'isolated': lambda: graphs.CSRGraph(np.zeros(71, np.int64), np.zeros(0, np.int64),
                                        np.zeros(0)),
    'clique31': lambda: _clique(31), 'clique32': lambda: _clique(32),
    'clique33': lambda: _clique(33), 'clique64': lambda: _clique(64),
    'clique65': lambda: _clique(65), 'clique200': lambda: _clique(200),
    'star512': lambda: _star(513), 'star513': lambda: _star(515), 'star3000': lambda: _star(3001),
    'path': lambda: _path(1000),
    'core': lambda: _core(6000, 150, 1),
    'messy': lambda: _messy(4),
    'rmat13': lambda: graphs.rmat(13, seed=3),
}


@pytest.mark.parametrize('order', ['id', 'jp'])
@pytest.mark.parametrize('name', sorted(CASES))
def test_equals_sequential_first_fit(name, order, monkeypatch):
    g = CASES[name]()
    monkeypatch.setenv('GRAPPOLO_B200_COLORING', order)
    monkeypatch.setenv('GRAPPOLO_B200_RECOLOR', '0')
    col, mc, _ = louvain.algoDistanceOneVertexColoringOpt(g, nThreads=8)
    expect = _first_fit(g, order == 'jp')
    assert np.array_equal(col, expect)
    assert mc == expect.max()


def test_too_many_colours_is_an_error():
    u, v = np.triu_indices(4097, k=1)
    with pytest.raises(_lib.GrappoloError) as e:
        louvain.algoDistanceOneVertexColoringOpt(_edges(4097, u, v), nThreads=1)
    assert e.value.code == 4  # GLV_ERR_COLORS

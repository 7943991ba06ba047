"""removeEdges with sorted rows on the device (rows merged from the kept edges'
two runs) against the oracle, entry for entry: integer and index work, so the
results must be identical."""
import numpy as np
import pytest

from grappolo_b200 import louvain

pytestmark = pytest.mark.gpu


def _edges(kind, n):
    rng = np.random.default_rng(n)
    if kind == 'both_ways':  # (u, v) and (v, u) both kept: ties in every row
        h, t = rng.integers(0, 40, n), rng.integers(0, 40, n)
        return 40, np.concatenate([h, t]), np.concatenate([t, h])
    if kind == 'late':  # repeats first, so that the late edges fill the holes
        h, t = rng.integers(0, 3, n), rng.integers(0, 3, n)
        a, b = rng.integers(0, 300, n), rng.integers(0, 300, n)
        return 300, np.concatenate([h, a, b]), np.concatenate([t, b, a])
    if kind == 'distinct':  # nothing dropped, no holes
        return 2 * n, np.arange(n), np.arange(n) + n
    if kind == 'loops':  # everything dropped
        h = rng.integers(0, 9, n)
        return 9, h, h
    if kind == 'star':  # one row holds an entry of every edge, from both runs
        leaf = rng.permutation(n) + 1
        hub = np.zeros(n, dtype=np.int64)
        flip = rng.random(n) < 0.5
        return n + 1, np.where(flip, leaf, hub), np.where(flip, hub, leaf)
    raise ValueError(kind)


@pytest.mark.parametrize('n', [1, 2, 255, 256, 257, 5000])
@pytest.mark.parametrize('kind', ['both_ways', 'late', 'distinct', 'loops', 'star'])
def test_merged_rows(oracle, kind, n):
    import torch
    nv, h, t = _edges(kind, n)
    w = np.arange(1, len(h) + 1) / 8.0  # a different weight for each place in the list
    rh, rt, rw, nge = oracle.remove_edges(nv, h, t, w)
    ptrs, sh, st, sw = oracle.sort_edges_undirected(nv, rh[:nge], rt[:nge], rw[:nge])
    _, ot, ow = oracle.sort_node_edges(nv, ptrs, sh, st, sw)
    g, nk = louvain.build_csr(nv, h, t, w, remove_edges=True, sort_rows=True)
    assert nk == nge and np.array_equal(g.ptr, ptrs[:nv + 1])
    assert np.array_equal(g.tail, ot) and np.array_equal(g.weight, ow)
    p, dt, dw = louvain.build_csr_device(nv, torch.tensor(h, device='cuda'),
                                         torch.tensor(t, device='cuda'),
                                         torch.tensor(w, device='cuda'), True, True)
    assert np.array_equal(p.cpu().numpy(), ptrs[:nv + 1])
    assert np.array_equal(dt.cpu().numpy(), ot) and np.array_equal(dw.cpu().numpy(), ow)

"""removeEdges with sorted rows on lists full of repeats in both directions: the
slots of late edges come from counts of dropped places, 128 at a time.  Against
the oracle, entry for entry."""
import numpy as np
import pytest

from grappolo_b200 import louvain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [2, 127, 128, 129, 255, 256, 257, 1024, 4097, 40000])
@pytest.mark.parametrize('distinct', [1, 3, 60, 1 << 20])  # edges drawn from at most this many
@pytest.mark.parametrize('order', ['shuffled', 'repeats_first', 'repeats_last'])
def test_repeats(oracle, n, distinct, order):
    import torch
    rng = np.random.default_rng(n + distinct)
    nv = max(2, n // 8)
    k = min(distinct, max(1, n // 2))
    h, t = rng.integers(0, nv, k), rng.integers(0, nv, k)
    e = rng.integers(0, k, n)
    if order != 'shuffled':  # every edge once, in one run before or after its repeats
        once = np.arange(k)
        e = np.concatenate([e, once] if order == 'repeats_first' else [once, e])
    flip = rng.random(e.size) < 0.5
    h, t = np.where(flip, t[e], h[e]), np.where(flip, h[e], t[e])
    w = np.arange(1, e.size + 1) / 8.0  # a different weight for each place in the list
    rh, rt, rw, nge = oracle.remove_edges(nv, h, t, w)
    ptrs, sh, st, sw = oracle.sort_edges_undirected(nv, rh[:nge], rt[:nge], rw[:nge])
    _, ot, ow = oracle.sort_node_edges(nv, ptrs, sh, st, sw)
    p, dt, dw = louvain.build_csr_device(nv, torch.tensor(h, device='cuda'),
                                         torch.tensor(t, device='cuda'),
                                         torch.tensor(w, device='cuda'), True, True)
    assert np.array_equal(p.cpu().numpy(), ptrs[:nv + 1])
    assert np.array_equal(dt.cpu().numpy(), ot) and np.array_equal(dw.cpu().numpy(), ow)


@pytest.mark.parametrize('n', [128 * 1024, 128 * 1024 + 1, 128 * 4096 - 1, 128 * 4096, 128 * 4096 + 1])
def test_counts_by_one_block_and_by_scan(oracle, n):
    """Lists on both sides of the limit of the counts that one block makes."""
    import torch
    rng = np.random.default_rng(n)
    nv = n // 16
    h, t = rng.integers(0, nv, n), rng.integers(0, nv, n)
    again = rng.integers(0, n, n // 3)
    put = rng.permutation(n)[:n // 3]
    h[put], t[put] = t[again], h[again]
    w = np.arange(1, n + 1) / 8.0
    rh, rt, rw, nge = oracle.remove_edges(nv, h, t, w)
    ptrs, sh, st, sw = oracle.sort_edges_undirected(nv, rh[:nge], rt[:nge], rw[:nge])
    _, ot, ow = oracle.sort_node_edges(nv, ptrs, sh, st, sw)
    p, dt, dw = louvain.build_csr_device(nv, torch.tensor(h, device='cuda'),
                                         torch.tensor(t, device='cuda'),
                                         torch.tensor(w, device='cuda'), True, True)
    assert np.array_equal(p.cpu().numpy(), ptrs[:nv + 1])
    assert np.array_equal(dt.cpu().numpy(), ot) and np.array_equal(dw.cpu().numpy(), ow)

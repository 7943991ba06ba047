"""Comparison on device labels that share memory: one array on both sides, and
two overlapping stretches of one array, with and without -1 entries (which the
two sides relabel differently), few ids and ids as many as vertices.  Integers
exact against the oracle on copies."""
import numpy as np
import pytest

from grappolo_b200 import louvain
from _golden import COMPARE_INTS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,ids', [(1, 1), (33, 4), (5000, 60), (5000, 5000), (60001, 700)])
@pytest.mark.parametrize('share', [0.0, 0.01, 0.3])  # of -1 entries
@pytest.mark.parametrize('base', [0, 1])
@pytest.mark.parametrize('shift', [0, 1, 7])
def test_shared_memory(oracle, n, ids, share, base, shift):
    import torch
    rng = np.random.default_rng(n + ids + shift)
    x = rng.integers(0, ids, n + shift) + base
    x[rng.random(n + shift) < share] = -1
    x[0] = x[shift] = base  # the base id is in use on both sides
    o, a, b = oracle.compare(x[:n], x[shift:])
    d = torch.tensor(x, device='cuda')
    st = louvain.compare_communities_device(d[:n], d[shift:])
    for k in COMPARE_INTS:
        assert st[k] == o[k], k
    want = x.copy()  # the relabelled arrays, the second side's values where they overlap
    want[:n] = a
    want[shift:] = b
    assert np.array_equal(d.cpu().numpy(), want)

"""Merge-path tiles at their edges: rows that end, start or span exactly at tile
boundaries, runs of empty rows, and levels of less than a tile.

glv_dev_modularity_static (which finds its tiles itself) and glv_modularity
against a numpy sum.  Weights are integers, so e_xx and the degrees are exact
in any order and compared exactly; Q within the parity tests' 1e-9.
"""
import ctypes as ct

import numpy as np
import pytest

from grappolo_b200 import _lib, graphs, louvain

pytestmark = pytest.mark.gpu

TILE = 4096


def _csr(degrees, seed):
    """A CSR with the given row lengths and random tails (modularity needs no symmetry)."""
    rng = np.random.default_rng(seed)
    ptr = np.zeros(len(degrees) + 1, dtype=np.int64)
    np.cumsum(degrees, out=ptr[1:])
    tail = rng.integers(0, len(degrees), ptr[-1])
    return graphs.CSRGraph(ptr, tail, rng.integers(1, 9, ptr[-1]).astype(np.float64))


CASES = {
    'one_entry': [1],
    'no_entries': [0] * 50,
    'row_ends_at_tile': [TILE - 1, 5, 7],
    'row_past_tile_by_one': [TILE, 5, 7],
    'entries_fill_tile': [TILE - 2, 0, 3],
    'empty_rows_fill_tiles': [3] + [0] * (2 * TILE) + [9, 0, 0],
    'hub_spans_tiles': [2, 5 * TILE + 17, 0, 4],
    'hub_ends_at_tile': [0, 3 * TILE - 2, 1],
    'mixed': list(np.random.default_rng(1).choice([0, 0, 1, 2, 31, 32, 33, 300, 5000], 3000)),
    'ones': [1] * (3 * TILE + 5),
}


@pytest.mark.parametrize('labels', ['few', 'many', 'none'])
@pytest.mark.parametrize('name', sorted(CASES))
def test_modularity(name, labels):
    import torch
    g = _csr(CASES[name], seed=3)
    nv = g.num_vertices
    rng = np.random.default_rng(4)
    C = rng.integers(0, {'few': min(3, nv), 'many': nv, 'none': nv}[labels], nv)
    if labels == 'none':
        C[rng.random(nv) < 0.4] = -1
    vdeg = np.bincount(g.heads(), weights=g.weight, minlength=nv)
    cdeg = np.zeros(nv)
    np.add.at(cdeg, C[C >= 0], vdeg[C >= 0])
    h = g.heads()
    same = (C[h] == C[g.tail]) & (C[h] >= 0)
    exx, a2 = float(g.weight[same].sum()), float((cdeg * cdeg).sum())
    k = 1.0 / max(float(g.weight.sum()), 1.0)
    d = dict(ptr=torch.from_numpy(g.ptr).cuda(),
             # (one spare entry: the entry point takes no NULL array)
             tail=torch.from_numpy(np.append(g.tail, 0).astype(np.int32)).cuda(),
             w=torch.from_numpy(np.append(g.weight, 0.0)).cuda(), C=torch.from_numpy(C.astype(np.int32)).cuda(),
             cdeg=torch.from_numpy(cdeg).cuda(),
             out=torch.full((3,), -7.0, dtype=torch.float64, device='cuda'))
    _lib.check(_lib.lib().glv_dev_modularity_static(
        nv, d['ptr'].data_ptr(), d['tail'].data_ptr(), d['w'].data_ptr(), d['C'].data_ptr(),
        d['cdeg'].data_ptr(), k, d['out'].data_ptr(),
        ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
    out = d['out'].cpu().numpy()
    assert out[1] == exx and out[2] == a2
    assert out[0] == pytest.approx(exx * k - a2 * k * k, rel=1e-9, abs=1e-15)
    if labels != 'none' and g.nnz:
        assert louvain.modularity(g, C) == pytest.approx(exx * k - a2 * k * k, rel=1e-9,
                                                         abs=1e-15)

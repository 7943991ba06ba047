"""glv_dev_modularity_static on a stretch of rows of a longer CSR: row offsets
that do not start at 0, over packed graphs with ids of their own.  Integer
weights, so e_xx and the degrees are exact in any order."""
import ctypes as ct

import numpy as np
import pytest

from grappolo_b200 import _lib

pytestmark = pytest.mark.gpu

TILE = 4096


@pytest.mark.parametrize('first', [1, 5, TILE, 3 * TILE + 7])  # entries before the stretch
@pytest.mark.parametrize('degrees', [[1], [0, 0, 0], [3, 0, 2 * TILE + 5, 1], [7] * 3000])
def test_offset_rows(degrees, first):
    import torch
    rng = np.random.default_rng(first + len(degrees))
    nv, after = len(degrees), 9
    ptr = first + np.concatenate([[0], np.cumsum(degrees)]).astype(np.int64)
    n = int(ptr[-1]) + after
    tail, w = rng.integers(0, nv, n), rng.integers(1, 9, n).astype(np.float64)
    C = rng.integers(0, min(nv, 3), nv)
    cdeg = rng.integers(0, 50, nv).astype(np.float64)
    head = np.repeat(np.arange(nv), degrees)
    t, x = tail[first:ptr[-1]], w[first:ptr[-1]]
    exx, a2 = float(x[C[head] == C[t]].sum()), float((cdeg * cdeg).sum())
    d = dict(ptr=torch.from_numpy(np.concatenate([[0, 0], ptr])).cuda(),
             tail=torch.from_numpy(tail.astype(np.int32)).cuda(), w=torch.from_numpy(w).cuda(),
             C=torch.from_numpy(C.astype(np.int32)).cuda(), cdeg=torch.from_numpy(cdeg).cuda(),
             out=torch.full((3,), -7.0, dtype=torch.float64, device='cuda'))
    _lib.check(_lib.lib().glv_dev_modularity_static(
        nv, d['ptr'].data_ptr() + 16, d['tail'].data_ptr(), d['w'].data_ptr(),
        d['C'].data_ptr(), d['cdeg'].data_ptr(), 0.5, d['out'].data_ptr(),
        ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
    out = d['out'].cpu().numpy()
    assert out[1] == exx and out[2] == a2
    assert out[0] == exx * 0.5 - a2 * 0.5 * 0.5

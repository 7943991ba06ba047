"""Fast mode's merging of colour classes does not follow the speed switches: with
the tuner off, on, or forced on small levels, a run takes the same steps and ends
in the same communities (id-order colouring and integer weights: nothing else
varies)."""
import numpy as np
import pytest

from grappolo_b200 import _lib, graphs, louvain

pytestmark = pytest.mark.gpu

TUNING = [{'GRAPPOLO_B200_AUTOTUNE': '0'}, {'GRAPPOLO_B200_AUTOTUNE': '1'},
          {'GRAPPOLO_B200_AUTOTUNE_MIN': '0'},
          {'GRAPPOLO_B200_AUTOTUNE_MIN': str(1 << 40)}]


@pytest.mark.parametrize('scale,factor', [(15, 16), (20, 16)])  # below and above 2^24 entries
def test_tuner_leaves_the_steps_alone(scale, factor, monkeypatch):
    import torch
    monkeypatch.setenv('GRAPPOLO_B200_COLORING', 'id')
    ptr, tail, w = graphs.rmat_device(scale, edge_factor=factor, seed=3, device='cuda')
    w = torch.ceil(w * 16)
    out = []
    for env in TUNING:
        with monkeypatch.context() as m:
            for k, v in env.items():
                m.setenv(k, v)
            C = torch.full((ptr.numel() - 1,), -1, dtype=torch.int32, device='cuda')
            st = louvain.run_multiphase_device(C.numel(), ptr.data_ptr(), tail.data_ptr(),
                                               w.data_ptr(), C.data_ptr(),
                                               mode=_lib.GLV_MODE_FAST)
            out.append((C.cpu().numpy(), st['final_modularity'], st['total_iterations']))
    for C, q, it in out[1:]:
        assert np.array_equal(C, out[0][0]) and q == out[0][1] and it == out[0][2]

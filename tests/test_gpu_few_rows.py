"""Levels whose steps have few rows (the sweep runs one block per SM) and levels
just past that line, in verify mode against the oracle."""
import numpy as np
import pytest

from grappolo_b200 import _lib, graphs, louvain

pytestmark = pytest.mark.gpu

LINE = 2 * 148 * 16 * 8  # a path of this many vertices: two classes, eight rows a warp


def _ring_of(n, reach):
    v = np.arange(n)
    return graphs.from_edges(n, [(int(i), int((i + k) % n)) for k in range(1, reach + 1)
                                 for i in v if n > 2 * reach])


@pytest.mark.parametrize('name,g', [
    ('pair', lambda: graphs.from_edges(2, [(0, 1)])),
    ('below', lambda: graphs.from_edges(LINE - 2, [(i, i + 1) for i in range(LINE - 3)])),
    ('at', lambda: graphs.from_edges(LINE, [(i, i + 1) for i in range(LINE - 1)])),
    ('past', lambda: graphs.from_edges(LINE + 2, [(i, i + 1) for i in range(LINE + 1)])),
    ('warp_rows', lambda: _ring_of(1200, 20)),      # 40 entries a row
    ('one_team_row', lambda: graphs.from_edges(
        400, [(0, i) for i in range(1, 200)] + [(i, i + 1) for i in range(1, 399)])),
], ids=lambda x: x if isinstance(x, str) else '')
def test_verify_equals_oracle(oracle, name, g):
    g = g()
    C, st = louvain.run_multiphase_csr(g, mode=_lib.GLV_MODE_VERIFY)
    Co, so, _ = oracle.run_multiphase_coloring(g)
    assert np.array_equal(C, Co), name
    assert st['phases'] == so['phases'] and st['total_iterations'] == so['total_iterations']

"""Without the reference's sources and without a build of them: the loader says so, and the
benchmark prints its lines all the same (the reference arm one that gives the reason)."""
import json

import pytest

import bench
from oracle import Reference, ReferenceMissing, lvoracle


@pytest.fixture
def no_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(lvoracle, 'HERE', str(tmp_path))
    monkeypatch.setattr(lvoracle, 'build', lambda ref=None: None)  # nothing to build from


@pytest.mark.parametrize('kind', [dict(), dict(fast=True), dict(patched_vbase=True)])
def test_loader_names_what_is_missing(no_reference, kind):
    with pytest.raises(ReferenceMissing, match='libgrappolo_ref'):
        Reference(**kind)


@pytest.mark.parametrize('workload', ['rmat', 'csr', 'compare'])
def test_reference_arm_prints_its_reason(no_reference, workload, monkeypatch, capsys):
    monkeypatch.setattr('sys.argv', ['bench.py', '--impl', 'reference', '--workload', workload])
    assert bench.main() == 0
    out = capsys.readouterr().out.strip().splitlines()
    assert len(out) == 1
    line = json.loads(out[0])
    assert line['impl'] == 'reference' and 'libgrappolo_ref_fast.so' in line['unavailable']


def test_baseline_is_the_reason(no_reference):
    assert set(bench.reference_unavailable()) == {'unavailable'}

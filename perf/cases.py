"""The work that this framework is timed on: multiphase Louvain in its modes, batches of graphs,
edge lists to CSR, modularity, comparison of communities and the move gate, each through its
public entry point.

Graphs are the families that the tests and bench.py generate (R-MAT, planted partitions, the
batched workload's mixed planted partitions).  Weights are one of

* ``unit``    1.0, as unweighted graph files load;
* ``count``   integers 1..16 (multiplicities), every sum exact;
* ``fixed``   multiples of 1/1024 in (0, 1]: not integers, so the engine takes its paths for
              fractional weights, but sums are still exact in any order;
* ``float``   uniform in (0, 1] with all 53 bits, only in verify mode, whose sums are ordered.

Fast mode's speculative colouring races, so two of its runs give different communities.  The runs
here use the documented id-order colouring (GRAPPOLO_B200_COLORING=id), which with the weights
above makes a run's communities reproducible.
"""
import ctypes as ct
import math
import os

import numpy as np
import torch

from grappolo_b200 import _lib, gate, graphs, louvain

os.environ.setdefault('GRAPPOLO_B200_COLORING', 'id')

DEV = 'cuda'
MODES = {'verify': _lib.GLV_MODE_VERIFY, 'fast': _lib.GLV_MODE_FAST,
         'learned': _lib.GLV_MODE_LEARNED}


def listed():
    return [
        # a small graph through the reference's own call, host graph in and communities out:
        # what one call costs at least
        dict(name='host_small_1200', kind='louvain', graph='mixed', nv=1201, block=60, mu=0.25,
             degree=14.0, weights='unit', mode='verify', coloring=True, host=True),
        # the plain parity workload: 100,000 vertices in blocks of 100, degree 16, host graph
        dict(name='host_planted_100k', kind='louvain', graph='mixed', nv=100000, block=100,
             mu=0.25, degree=16.0, weights='unit', mode='verify', coloring=True, host=True),
        # verify mode on real-valued weights: ordered sums, one launch sequence per colour class
        dict(name='verify_float_rmat15', kind='louvain', graph='rmat', scale=15, edge_factor=16,
             weights='float', mode='verify', coloring=True, host=False),
        # verify mode on a skewed graph with integral weights, resident on the device
        dict(name='verify_rmat18', kind='louvain', graph='rmat', scale=18, edge_factor=16,
             weights='count', mode='verify', coloring=True, host=False),
        # fast mode on skewed graphs with fractional weights: an ordinary one and the largest
        dict(name='fast_rmat20', kind='louvain', graph='rmat', scale=20, edge_factor=16,
             weights='fixed', mode='fast', coloring=True, host=False),
        dict(name='fast_rmat22', kind='louvain', graph='rmat', scale=22, edge_factor=14,
             weights='fixed', mode='fast', coloring=True, host=False),
        # the basic (Jacobi) driver in fast mode
        dict(name='basic_rmat22', kind='louvain', graph='rmat', scale=22, edge_factor=16,
             weights='fixed', mode='fast', coloring=False, host=False),
        # learned mode: the move gate inside the sweeps
        dict(name='learned_mixed_1m', kind='louvain', graph='mixed', nv=1000003, block=150, mu=0.4,
             degree=20.0, weights='count', mode='learned', coloring=True, host=False),
        # many graphs of the batched workload in one run
        dict(name='batch_200', kind='batch', count=200, spec_seed=3, mode='fast', coloring=True),
        # a raw R-MAT edge list (repeats, self-loops) to a sorted CSR
        dict(name='csr_rmat22', kind='csr', scale=22, edge_factor=16, drop=123, remove=True,
             sort=True),
        # modularity of an assignment, allocation-free, on a skewed graph
        dict(name='modularity_rmat22', kind='modularity', graph='rmat', scale=22, edge_factor=16,
             weights='float', block=64),
        # comparing an output with the truth
        dict(name='compare_20m', kind='compare', n=20000003, block=150, noise=0.2),
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def _draw_graph(rng, scale_hi, nv_hi):
    if rng.random() < 0.5:
        return dict(graph='rmat', scale=rng.randint(12, scale_hi), edge_factor=rng.randint(5, 16))
    return dict(graph='mixed', nv=_log_int(rng, 700, nv_hi) | 1, block=_log_int(rng, 20, 600),
                mu=round(rng.uniform(0.1, 0.55), 3), degree=round(rng.uniform(6.0, 32.0), 2))


def draw(rng):
    kind = rng.choice(['louvain'] * 5 + ['batch', 'csr', 'modularity', 'compare'])
    if kind == 'batch':
        return dict(kind=kind, count=_log_int(rng, 12, 180), spec_seed=rng.randint(4, 10000),
                    mode=rng.choice(['verify', 'fast']), coloring=rng.random() < 0.7)
    if kind == 'csr':
        return dict(kind=kind, scale=rng.randint(12, 22), edge_factor=rng.randint(5, 16),
                    drop=rng.randint(0, 999), remove=rng.random() < 0.7, sort=rng.random() < 0.7)
    if kind == 'modularity':
        return dict(_draw_graph(rng, 22, 2000000), kind=kind,
                    weights=rng.choice(['unit', 'float']), block=_log_int(rng, 8, 4000))
    if kind == 'compare':
        return dict(kind=kind, n=_log_int(rng, 3000, 19000000) | 1, block=_log_int(rng, 20, 5000),
                    noise=round(rng.uniform(0.05, 0.5), 3))
    mode = rng.choice(['verify', 'verify', 'fast', 'fast', 'learned'])
    coloring = mode == 'learned' or rng.random() < 0.75
    weights = rng.choice({'verify': ['unit', 'count', 'float'], 'fast': ['unit', 'count', 'fixed'],
                          'learned': ['count', 'fixed']}[mode])
    if weights == 'float':
        shape = _draw_graph(rng, 15, 60000)
    elif mode == 'verify':
        shape = _draw_graph(rng, 18, 1000000)
    else:
        shape = _draw_graph(rng, 21, 2000000)
    host = mode != 'learned' and rng.random() < 0.3
    return dict(shape, kind=kind, weights=weights, mode=mode, coloring=coloring, host=host)


def _make_graph(case, seed):
    """(ptr int64, tail int32, weight float64) on the device, rows sorted by tail."""
    kind = case.get('weights', 'unit')
    if case['graph'] == 'rmat':
        ptr, tail, w = graphs.rmat_device(case['scale'], edge_factor=case['edge_factor'],
                                          seed=seed, device=DEV)
    else:
        spec = np.array([[case['nv'], min(case['block'], case['nv']), case['mu'],
                          case['degree']]])
        _, ptr, tail, w = graphs.planted_batch_device(spec, seed=seed, device=DEV)
        if kind != 'unit':
            # one uniform value per undirected edge, from a hash of its ends
            nv = ptr.numel() - 1
            row = torch.repeat_interleave(torch.arange(nv, device=DEV), ptr[1:] - ptr[:-1])
            t = tail.to(torch.int64)
            h = torch.minimum(row, t) * nv + torch.maximum(row, t) + (seed % 65521)
            h = (h ^ (h >> 31)) * 0x7FB5D329728EA185
            h = (h ^ (h >> 27)) * 0x1B03738712FAD5C9
            w = 1.0 - ((h >> 11) & ((1 << 53) - 1)).to(torch.float64) * 2.0 ** -53
    if kind == 'unit':
        w = torch.ones_like(w)
    elif kind == 'count':
        w = torch.ceil(w * 16.0)
    elif kind == 'fixed':
        w = torch.ceil(w * 1024.0) / 1024.0
    return ptr, tail, w


def _labels(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    n = case['n']
    truth = torch.arange(n, device=DEV) // case['block']
    k = int(truth[-1]) + 1
    out = truth.clone()
    moved = torch.rand(n, generator=gen, device=DEV) < case['noise']
    moved[0] = False  # label 0 stays in use on both sides: 0-based ids
    out[moved] = torch.randint(0, k, (int(moved.sum()),), generator=gen, device=DEV)
    order = torch.randperm(n - 1, generator=gen, device=DEV) + 1
    return (torch.cat([truth[:1], truth[order]]).contiguous(),
            torch.cat([out[:1], out[order]]).contiguous())


def prepare(case, seed):
    kind = case['kind']
    s = dict(case=case)
    if kind == 'louvain':
        if case['mode'] == 'learned':
            gate.set_gate(*gate.load_default())
        ptr, tail, w = _make_graph(case, seed)
        if case['host']:
            csr = graphs.CSRGraph(ptr.cpu().numpy(), tail.cpu().numpy().astype(np.int64),
                                  w.cpu().numpy())
            s['G'] = louvain.Graph(csr)
        else:
            s.update(ptr=ptr, tail=tail, w=w,
                     C=torch.full((ptr.numel() - 1,), -1, dtype=torch.int32, device=DEV))
    elif kind == 'batch':
        specs = graphs.batch_specs(case['count'], seed=case['spec_seed'])
        voff, ptr, tail, w = graphs.planted_batch_device(specs, seed=seed, device=DEV)
        s.update(voff=voff, ptr=ptr, tail=tail, w=w,
                 C=torch.full((ptr.numel() - 1,), -1, dtype=torch.int32, device=DEV))
    elif kind == 'csr':
        head, tail, w = graphs.rmat_edges_device(case['scale'], edge_factor=case['edge_factor'],
                                                 seed=seed, device=DEV)
        n = head.numel() - case['drop']
        nv = 1 << case['scale']
        s.update(nv=nv, head=head[:n].contiguous(), tail=tail[:n].contiguous(),
                 w=w[:n].contiguous(), ptr=torch.zeros(nv + 1, dtype=torch.int64, device=DEV),
                 out_tail=torch.zeros(2 * n, dtype=torch.int32, device=DEV),
                 out_w=torch.zeros(2 * n, dtype=torch.float64, device=DEV))
    elif kind == 'modularity':
        ptr, tail, w = _make_graph(case, seed)
        nv = ptr.numel() - 1
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed + 1)
        # an assignment like a level's result: communities of `block` vertices on average,
        # isolated vertices in none
        C = torch.randint(0, max(1, nv // case['block']), (nv,), generator=gen, device=DEV)
        deg = ptr[1:] - ptr[:-1]
        cum = torch.zeros(w.numel() + 1, dtype=torch.float64, device=DEV)
        torch.cumsum(w, 0, out=cum[1:])
        vdeg = cum[ptr[1:]] - cum[ptr[:-1]]
        cdeg = torch.zeros(nv, dtype=torch.float64, device=DEV)
        cdeg.index_put_((C,), torch.where(deg > 0, vdeg, torch.zeros_like(vdeg)), accumulate=True)
        C = torch.where(deg > 0, C, torch.full_like(C, -1)).to(torch.int32)
        s.update(ptr=ptr, tail=tail, w=w, C=C, cdeg=cdeg, constant=1.0 / float(cum[-1]),
                 out=torch.zeros(3, dtype=torch.float64, device=DEV))
    else:
        s['truth'], s['output'] = _labels(case, seed)
    return s


def _result(C, st):
    return {'C': C, 'modularity': float(st['final_modularity']), 'phases': int(st['phases']),
            'iterations': int(st['total_iterations']), 'clusters': int(st['final_clusters'])}


def run(s):
    case = s['case']
    kind = case['kind']
    if kind == 'louvain' and case['host']:
        threads = 1 if case['mode'] == 'verify' else 16
        call = louvain.runMultiPhaseColoring if case['coloring'] else louvain.runMultiPhaseBasic
        return _result(*call(s['G'], numThreads=threads, stats=True))
    if kind == 'louvain':
        st = louvain.run_multiphase_device(
            s['ptr'].numel() - 1, s['ptr'].data_ptr(), s['tail'].data_ptr(), s['w'].data_ptr(),
            s['C'].data_ptr(), coloring=case['coloring'], mode=MODES[case['mode']])
        return _result(s['C'], st)
    if kind == 'batch':
        st = louvain.run_batch_device(
            s['voff'], s['ptr'].data_ptr(), s['tail'].data_ptr(), s['w'].data_ptr(),
            s['C'].data_ptr(), coloring=case['coloring'], mode=MODES[case['mode']])
        return {'C': s['C'], 'modularity': st['final_modularity'], 'phases': st['phases'],
                'iterations': st['iterations'], 'clusters': st['clusters']}
    if kind == 'csr':
        flags = (_lib.GLV_CSR_REMOVE_EDGES if case['remove'] else 0) | \
            (_lib.GLV_CSR_SORT_ROWS if case['sort'] else 0)
        nnz = ct.c_long(0)
        _lib.check(_lib.lib().glv_dev_build_csr(
            s['nv'], s['head'].numel(), s['head'].data_ptr(), s['tail'].data_ptr(),
            s['w'].data_ptr(), flags, s['ptr'].data_ptr(), s['out_tail'].data_ptr(),
            s['out_w'].data_ptr(), ct.byref(nnz),
            ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {'ptr': s['ptr'], 'tail': s['out_tail'], 'weight': s['out_w'], 'nnz': nnz.value}
    if kind == 'modularity':
        _lib.check(_lib.lib().glv_dev_modularity_static(
            s['ptr'].numel() - 1, s['ptr'].data_ptr(), s['tail'].data_ptr(), s['w'].data_ptr(),
            s['C'].data_ptr(), s['cdeg'].data_ptr(), s['constant'], s['out'].data_ptr(),
            ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return s['out']
    return louvain.compare_communities_device(s['truth'], s['output'],
                                              torch.cuda.current_stream().cuda_stream)


def _graph_sizes(case):
    """(vertices, CSR entries) that the graph's parameters ask for; repeats and self-loops, which
    the generators drop, are left out at their share in R-MAT lists of these sizes."""
    if case['graph'] == 'rmat':
        nv = 1 << case['scale']
        return nv, int(1.85 * case['edge_factor'] * nv)
    return case['nv'], int(0.95 * case['degree'] * case['nv'])


def work(case):
    """Every input once and every output once: a run cannot do without reading its graph (12 B
    per entry, 8 B per vertex) and writing the communities (4 B; 8 B in host arrays)."""
    kind = case['kind']
    if kind == 'louvain':
        nv, nnz = _graph_sizes(case)
        if case['host']:  # 24 B records
            return {'bytes': 24 * nnz + 16 * nv, 'flops': 2 * nnz}
        return {'bytes': 12 * nnz + 12 * nv, 'flops': 2 * nnz}
    if kind == 'batch':
        specs = graphs.batch_specs(case['count'], seed=case['spec_seed'])
        nv, nnz = int(specs[:, 0].sum()), int(0.95 * (specs[:, 0] * specs[:, 3]).sum())
        return {'bytes': 12 * nnz + 12 * nv, 'flops': 2 * nnz}
    if kind == 'csr':
        ne = (case['edge_factor'] << case['scale']) - case['drop']
        kept = 0.93 * ne if case['remove'] else ne
        return {'bytes': int(24 * ne + 24 * kept + (8 << case['scale'])), 'flops': 0}
    if kind == 'modularity':
        nv, nnz = _graph_sizes(case)
        return {'bytes': 12 * nnz + 20 * nv, 'flops': nnz}
    return {'bytes': 16 * case['n'], 'flops': 0}


def exact(case, seed):
    """Modularity and the comparison's ratios in 64 bits.  The other cases' floating outputs
    depend on the run's own decisions (modularity) or are moved, not computed (CSR weights)."""
    if case['kind'] == 'modularity':
        s = prepare(case, seed)
        nv = s['ptr'].numel() - 1
        row = torch.repeat_interleave(torch.arange(nv, device=DEV), s['ptr'][1:] - s['ptr'][:-1])
        c = s['C'][row]
        same = (c == s['C'][s['tail'].to(torch.int64)]) & (c >= 0)
        exx = float(s['w'][same].sum())
        a2 = float((s['cdeg'] * s['cdeg']).sum())
        k = s['constant']
        return np.array([exx * k - a2 * k * k, exx, a2])
    if case['kind'] == 'compare':
        truth, out = (x.cpu().numpy() for x in _labels(case, seed))

        def pairs(counts):
            counts = counts.astype(object) if counts.dtype == object else counts.astype(np.int64)
            return int((counts * (counts - 1) // 2).sum())

        def gini(counts):
            x = np.sort(counts).astype(np.float64)
            n = x.size
            return None if n == 0 else float(
                (2.0 * (np.arange(1, n + 1) * x).sum()) / (n * x.sum()) - (n + 1.0) / n)

        ct1, ct2 = np.bincount(truth), np.bincount(out)
        both = np.unique(truth * (int(out.max()) + 1) + out, return_counts=True)[1]
        ss, p1, p2 = pairs(both), pairs(ct1), pairs(ct2)
        precision, recall = ss / p2, ss / p1
        return {'precision': precision, 'recall': recall,
                'f_score': 2.0 * precision * recall / (precision + recall),
                'gini1': gini(ct1), 'gini2': gini(ct2)}
    return None

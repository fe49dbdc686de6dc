"""The captured sweeps and their split rows: rows of many chunks, whose chunk sums
a warp or (past 2,048 of them) a whole CTA adds, in the sweeps, with weights, in
the centralities and in the adjoint, whose split rows are the out-rows; no split
rows at all; and a graph between the sizes of one launch and of source blocks."""
import os

import numpy as np
import pytest

from networkit_b200 import _capi, generators
from networkit_b200.graph import InCSR

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 1
# 64-arc chunks: 2,048 and 2,049 sums, more than a pass of a CTA (256 x 16), rows of
# a warp and of a thread in the same CTA of the fix-up; two rows for a CTA, and three
# (which its warps take)
LENGTHS = {"cta": [300_001, 131_073, 131_072, 131_071, 20_000, 1_025, 1_024, 65, 64, 7],
           "warps": [300_001, 131_073, 262_145, 131_072, 20_000, 1_025, 1_024, 65, 64, 7]}


@pytest.fixture(scope="module", params=sorted(LENGTHS))
def graph(request):
    """Nodes with these in-degrees, and others with these out-degrees."""
    lengths = LENGTHS[request.param]
    rng = np.random.default_rng(3)
    n, k = 50_000, len(lengths)
    hub = np.repeat(np.arange(k), lengths)
    src = np.concatenate([rng.integers(0, n, hub.size), hub + k, rng.integers(0, n, 200_000)])
    dst = np.concatenate([hub, rng.integers(2 * k, n, hub.size), rng.integers(2 * k, n, 200_000)])
    order = np.argsort(dst, kind="stable")
    ptr = np.concatenate([[0], np.cumsum(np.bincount(dst, minlength=n))]).astype(np.uint64)
    out = np.bincount(src, minlength=n)
    csr = InCSR(n, n, ptr, src[order].astype(np.uint32), None, out.astype(np.float64),
                out.astype(np.uint32), None, True)
    assert np.diff(ptr.astype(np.int64))[:k].tolist() == lengths
    return csr


@pytest.mark.parametrize("weighted", [False, True])
def test_split_rows_match_oracle(oracle_mod, graph, weighted):
    csr = generators.with_uniform_weights(graph, seed=2) if weighted else graph
    dg = _capi.DeviceGraph(csr, hot_tier_kb=0)
    o = oracle_mod.pagerank(csr, tol=1e-11, norm=0, distribute_sinks=True, nthreads=THREADS)
    p = dg.params(0.85, 1e-11, 0, False, True, _capi.NKG_PREC_FP64, 5000)
    s, it, _, _ = dg.run(p)
    assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-10
    np.testing.assert_array_equal(dg.run(p)[0], s)
    p.precision = _capi.NKG_PREC_FP32_REFINE
    # both stop at a residual of 1e-11, at most 1e-11 / (1 - 0.85) from the fixed point
    assert np.abs(dg.run(p)[0] - o.scores).sum() <= 2e-10
    p32 = dg.params(0.85, 0.0, 0, False, True, _capi.NKG_PREC_FP32, 60)
    # FP32 scores of unit mass: a few roundings of 2^-24 each
    assert np.abs(dg.run(p32)[0] - o.scores).sum() <= 1e-6


def test_split_rows_of_the_centralities_match_oracle(oracle_mod, graph):
    dg = _capi.DeviceGraph(graph)
    s, it, _ = dg.eigenvector(1e-9)
    o, _ = oracle_mod.eigenvector(graph, -1.0, max_iterations=it)
    assert np.abs(s - o).sum() <= 1e-10 * np.abs(o).sum()


def test_split_rows_of_the_adjoint(graph):
    csr = generators.with_uniform_weights(graph, seed=2)
    dg = _capi.DeviceGraph(csr)
    p = dg.params(0.85, 1e-12, 0, False, True, _capi.NKG_PREC_FP64, _capi.UINT64_MAX)
    s = dg.run(p)[0]
    g = np.random.default_rng(0).standard_normal(csr.z)
    gw, gt, _, _ = dg.adjoint(p, s, g)
    p.precision, p.tol = _capi.NKG_PREC_FP32_REFINE, 1e-11
    gw2, gt2, _, _ = dg.adjoint(p, s, g)
    assert np.abs(gw - gw2).max() <= 1e-9 * np.abs(gw).max()
    assert np.abs(gt - gt2).max() <= 1e-9 * np.abs(gt).max()
    # the arcs of the largest gradients, by central differences of the forward run
    f = dg.params(0.85, 0.0, 0, False, True, _capi.NKG_PREC_FP64, 250)
    for e in np.argsort(-np.abs(gw))[[0, 5]]:
        vals = []
        for h in (1e-4, -1e-4):
            w = csr.in_w.copy()
            w[e] += h
            dg.set_weights(w)
            vals.append(float(g @ dg.run(f)[0]))
        assert abs((vals[0] - vals[1]) / 2e-4 - gw[e]) <= 1e-4 * abs(gw[e])


@pytest.mark.parametrize("n, deg", [(100_000, 10), (400_000, 8)])
def test_captured_sweeps_without_split_rows(oracle_mod, n, deg):
    """Few enough work units that the sweep's last CTA closes every iteration (one
    launch a sweep), and more than 8,192, so that a fix-up without split rows adds
    the units' partials (two launches)."""
    csr = generators.erdos_renyi(n, deg / (n - 1), seed=5)
    dg = _capi.DeviceGraph(csr, hot_tier_kb=0)
    assert dg.info()["split_rows"] == 0
    for distribute in (False, True):
        o = oracle_mod.pagerank(csr, tol=1e-10, norm=0, distribute_sinks=distribute)
        p = dg.params(0.85, 1e-10, 0, False, distribute, _capi.NKG_PREC_FP64, 5000)
        s, it, _, st = dg.run(p)
        assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-10
        np.testing.assert_array_equal(dg.run(p)[0], s)
        # batches of 2, 4, 8, 8, ... captured graphs of 8 sweeps, three launches beside
        sweeps = [16, 48, 112, 176, 240]
        took = next(k for k in sweeps if k >= it)
        assert st["kernel_launches"] == took * (1 if n == 100_000 else 2) + 3


def test_graph_past_one_launch_and_below_source_blocks(oracle_mod):
    csr = generators.rmat_directed(21, 16, seed=4)
    assert 20 << 20 < csr.arcs < 60 << 20
    dg = _capi.DeviceGraph(csr)
    o = oracle_mod.pagerank(csr, tol=1e-10, norm=0, distribute_sinks=True, nthreads=THREADS)
    p = dg.params(0.85, 1e-10, 0, False, True, _capi.NKG_PREC_FP64, 5000)
    s, it, _, st = dg.run(p)
    assert st["kernel_launches"] > 1
    assert st["bytes_per_sweep_fp64"] == 4 * csr.arcs + 4 * (csr.n + 1) + 28 * csr.n  # no blocks
    assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-10
    p.precision = _capi.NKG_PREC_FP32_REFINE
    assert np.abs(dg.run(p)[0] - o.scores).sum() <= 2e-9
    p32 = dg.params(0.85, 0.0, 0, False, True, _capi.NKG_PREC_FP32, 60)
    assert np.abs(dg.run(p32)[0] - o.scores).sum() <= 2e-6


@pytest.mark.parametrize("n,reach,whole", [(150_000, 150, False), (200_000, 150, True)])
def test_long_rows_of_local_ids(oracle_mod, n, reach, whole):
    """Rows of 80 arcs to nearby ids, 12M and 16M arcs: captured sweeps, not one
    launch, and with a row for nearly every resident lane the rows stay whole
    although they are longer than a chunk of 64."""
    rng = np.random.default_rng(n)
    lens = rng.integers(70, 91, n)
    dst = np.repeat(np.arange(n), lens)
    src = ((dst + rng.integers(1, reach, dst.size)) % n).astype(np.uint32)
    out = np.bincount(src, minlength=n)
    csr = InCSR(n, n, np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64), src, None,
                out.astype(np.float64), out.astype(np.uint32), None, True)
    dg = _capi.DeviceGraph(csr)
    info = dg.info()
    assert info["row_order"] == 1 and (info["split_rows"] == 0) == whole
    o = oracle_mod.pagerank(csr, tol=1e-10, norm=0, distribute_sinks=True, nthreads=THREADS)
    p = dg.params(0.85, 1e-10, 0, False, True, _capi.NKG_PREC_FP64, 5000)
    s, it, _, st = dg.run(p)
    assert st["kernel_launches"] > 1
    assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-10
    s2 = _capi.DeviceGraph(csr, row_order=0).run(p)[0]  # one launch
    assert np.abs(s2 - o.scores).sum() <= 1e-10

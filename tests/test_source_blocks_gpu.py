"""Layouts whose long rows are grouped by source blocks (unweighted graphs of 60 Mi
arcs and more whose leading sources are gathered most) against the oracle: the
plain and the centrality sweeps, the FP32 forms, every order of rows and arcs, a
last block of few ids; and on graphs of that size what has no blocks: weights and
their gradients, and personalised PageRank, which reads the CSR itself."""
import os

import numpy as np
import pytest

from networkit_b200 import _capi, generators
from networkit_b200.graph import InCSR

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 1


def blocks_of(dg, csr):
    """Whether the layout has source blocks: a sweep's bytes count their arcs as
    16-bit ids."""
    st = dg.run(dg.params(0.85, 0.0, 0, False, False, _capi.NKG_PREC_FP64, 1))[3]
    return st["bytes_per_sweep_fp64"] < 4 * csr.arcs + 4 * (csr.n + 1) + 28 * csr.n


@pytest.fixture(scope="module")
def rmat():
    """R-MAT 22: large enough for source blocks, hubs of tens of thousands of
    arcs (partitioned by a whole CTA)."""
    csr = generators.rmat_directed(22, 18, seed=7)
    dg = _capi.DeviceGraph(csr)
    assert csr.arcs >= 60 << 20  # smaller graphs have none
    assert blocks_of(dg, csr)
    return csr, dg


@pytest.mark.parametrize("norm,distribute", [(0, False), (1, True)])
def test_blocked_sweeps_match_oracle(oracle_mod, rmat, norm, distribute):
    csr, dg = rmat
    tol = 1e-10 if norm == 0 else 1e-12
    o = oracle_mod.pagerank(csr, tol=tol, norm=norm, distribute_sinks=distribute, nthreads=THREADS)
    p = dg.params(0.85, tol, norm, False, distribute, _capi.NKG_PREC_FP64, _capi.UINT64_MAX)
    s, it, _, _ = dg.run(p)
    assert abs(it - o.iterations) <= 1
    assert np.abs(s - o.scores).sum() <= 1e-10
    s2, it2, _, _ = dg.run(p)
    np.testing.assert_array_equal(s, s2)
    assert it == it2
    if norm == 0:
        p = dg.params(0.85, tol, norm, False, distribute, _capi.NKG_PREC_FP32_REFINE, 10000)
        s, _, _, _ = dg.run(p)
        # both stop at a residual of 1e-10, at most 1e-10 / (1 - 0.85) from the fixed point
        assert np.abs(s - o.scores).sum() <= 2e-9


def test_fp32_rows_of_many_segments_round_like_their_epilogue(rmat):
    """Rows of 17 to 128 chunk sums: added in FP32 (four lanes, then across them)
    the sums cost 0.91 in the unit below. Left are the chunks' own sums, whose
    errors average out over dozens of chunks, and the four roundings of a row's
    epilogue and output, each uniform in one unit times a mantissa of 0.72 on
    average: sqrt(4 / 3) * 0.72."""
    csr, dg = rmat
    rows = np.diff(csr.in_ptr.astype(np.int64))
    rows = (rows >= 8000) & (rows < 16000)
    assert rows.sum() > 200
    s32, s64 = (dg.run(dg.params(0.85, 0.0, 0, False, False, prec, 5))[0]
                for prec in (_capi.NKG_PREC_FP32, _capi.NKG_PREC_FP64))
    rel = (s32 / s64 - 1) * 2.0 ** 24
    rel = rel[rows] - np.median(rel)  # the normalisation's factor is every row's
    assert np.sqrt((rel * rel).mean()) <= np.sqrt(4 / 3) * 0.72


@pytest.fixture(scope="module")
def rmat_scores(oracle_mod, rmat):
    return oracle_mod.pagerank(rmat[0], tol=1e-10, norm=0, distribute_sinks=True, nthreads=THREADS)


def close_to(dg, o):
    """FP64, FP32 and refined runs against FP64 scores of the oracle (tol 1e-10)."""
    p = dg.params(0.85, 1e-10, 0, False, True, _capi.NKG_PREC_FP64, 5000)
    s, it, _, _ = dg.run(p)
    assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-10
    p32 = dg.params(0.85, 0.0, 0, False, True, _capi.NKG_PREC_FP32, 60)
    # FP32 scores of unit mass: a few roundings of 2^-24 each
    assert np.abs(dg.run(p32)[0] - o.scores).sum() <= 2e-6
    p.precision = _capi.NKG_PREC_FP32_REFINE
    # both stop at a residual of 1e-10, at most 1e-10 / (1 - 0.85) from the fixed point
    assert np.abs(dg.run(p)[0] - o.scores).sum() <= 2e-9


@pytest.mark.parametrize("options", [dict(row_order=1), dict(row_order=0), dict(arc_order=1),
                                     dict(hot_tier_kb=64), dict(hot_tier_kb=200),
                                     dict(sweep_shape=2)], ids=str)
def test_every_layout_option_with_blocks(rmat, rmat_scores, options):
    dg = _capi.DeviceGraph(rmat[0], **options)
    assert blocks_of(dg, rmat[0])
    close_to(dg, rmat_scores)


@pytest.mark.parametrize("n", [3 * 24576 + 1, 2 * 24576 + 3, 24576 + 24575])
def test_a_last_block_of_few_ids(oracle_mod, n):
    """Dense graphs whose last block of 24,576 sources has one id, three (no whole
    16 bytes) and all but one."""
    rng = np.random.default_rng(n)
    arcs = 64 << 20
    lens = rng.multinomial(arcs, rng.dirichlet(np.full(n, 3.0)))
    src = rng.integers(0, n, arcs, dtype=np.uint32)
    out = np.bincount(src, minlength=n)
    csr = InCSR(n, n, np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64), src, None,
                out.astype(np.float64), out.astype(np.uint32), None, True)
    dg = _capi.DeviceGraph(csr)
    assert blocks_of(dg, csr)
    close_to(dg, oracle_mod.pagerank(csr, tol=1e-10, norm=0, distribute_sinks=True,
                                     nthreads=THREADS))


def test_blocked_centralities_match_oracle(oracle_mod, rmat):
    csr, dg = rmat
    s, it, _ = dg.eigenvector(1e-9)
    o, _ = oracle_mod.eigenvector(csr, -1.0, max_iterations=it)
    assert np.abs(s - o).sum() <= 1e-10 * np.abs(o).sum()
    s, it, _ = dg.katz(0.0, 0.1, 1e-8, 0)
    o, _ = oracle_mod.katz(csr.z, csr.in_ptr, csr.in_col, alpha=0.0, beta=0.1, tol=-1.0,
                           max_degree=int(csr.outdeg.max()), max_iterations=it)
    # scores of unit 2-norm over 2^22 nodes: L1 up to 2048
    assert np.abs(s - o).sum() <= 1e-10 * np.abs(o).sum()


def test_ppr_columns_match_the_fp64_run_with_blocks(rmat):
    csr, dg = rmat
    seeds = np.array([5, 1 << 21, 77], np.uint32)
    p = dg.params(0.85, 1e-8, 0, False, True, _capi.NKG_PREC_FP32, 300)
    got, _, _ = dg.ppr(seeds, p)
    p64 = dg.params(0.85, 1e-12, 0, False, True, _capi.NKG_PREC_FP64, 2000)
    for j, u in enumerate(seeds):
        t = np.zeros(csr.z)
        t[u] = 1.0
        assert np.abs(got[j] - dg.run(p64, t)[0]).sum() <= 1e-6


def test_weighted_graph_of_that_size_and_its_gradients(oracle_mod, rmat):
    a = generators.with_uniform_weights(rmat[0], seed=3)
    b = generators.with_uniform_weights(rmat[0], seed=4)
    dg, ref = _capi.DeviceGraph(a), _capi.DeviceGraph(b)
    p = dg.params(0.85, 1e-10, 0, False, True, _capi.NKG_PREC_FP64, 500)
    dg.run(p)
    dg.set_weights(b.in_w, b.wdeg)
    got, want = dg.run(p)[0], ref.run(p)[0]
    np.testing.assert_array_equal(got, want)
    o = oracle_mod.pagerank(b, tol=1e-10, norm=0, distribute_sinks=True, nthreads=THREADS)
    assert np.abs(want - o.scores).sum() <= 1e-10
    g = np.random.default_rng(0).standard_normal(a.z)
    bwd = dg.params(0.85, 1e-11, 0, False, True, _capi.NKG_PREC_FP32_REFINE, _capi.UINT64_MAX)
    b64 = dg.params(0.85, 1e-12, 0, False, True, _capi.NKG_PREC_FP64, _capi.UINT64_MAX)
    gw, gt, _, _ = dg.adjoint(bwd, want, g)
    gw2, gt2, _, _ = ref.adjoint(b64, want, g)
    assert np.abs(gw - gw2).max() <= 1e-9 * np.abs(gw2).max()
    assert np.abs(gt - gt2).max() <= 1e-9 * np.abs(gt2).max()
    # central differences of the FP64 forward on the arcs of the largest gradients
    for e in np.argsort(-np.abs(gw2))[[0, 3]]:
        vals = []
        for h in (1e-4, -1e-4):
            w = b.in_w.copy()
            w[e] += h
            dg.set_weights(w)
            vals.append(float(g @ dg.run(dg.params(0.85, 0.0, 0, False, True, 0, 250))[0]))
        fd = (vals[0] - vals[1]) / 2e-4
        assert abs(fd - gw2[e]) <= 1e-4 * abs(gw2[e])


def test_blocks_are_left_out_where_memory_is_short(fail_alloc, rmat):
    """Every allocation of the graph's creation fails in turn: those of the blocks
    leave a graph without them, the others are the call's error."""
    csr, dg = rmat
    p = dg.params(0.85, 1e-9, 0, False, True, _capi.NKG_PREC_FP64, 500)
    want, want_it = dg.run(p)[:2]
    plain = 0
    for k in range(300):
        fail_alloc(k)
        try:
            h = _capi.DeviceGraph(csr)
        except _capi.NkgError as e:
            assert e.code == _capi.NKG_ERR_OOM
            continue
        if fail_alloc(-1) >= 0:
            break  # fewer than k + 1 allocations
        plain += 1
        assert not blocks_of(h, csr)
        s, it = h.run(p)[:2]
        # another order of summation of the same sweeps
        assert it == want_it and np.abs(s - want).sum() <= 1e-11
    assert plain >= 10 and k < 299

"""The one-launch run of small unweighted graphs against the oracle, at the
sizes where its row classes, hub rows, task counts and launches change."""
import numpy as np
import pytest

from networkit_b200 import _capi
from networkit_b200.graph import in_csr_from_edges

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def bar(z):
    """L1 distance two FP64 runs of the same sweeps may have. The oracle adds the
    z scores (and residual terms) one after the other, an error of up to
    z eps / 2 of a unit-mass sum, which the normalisation spreads over all
    scores; the row sums add a few eps per sweep."""
    return 1e-13 + z * EPS


def graph_of_rows(lengths, n, seed):
    """Directed graph on n nodes whose node i < len(lengths) has lengths[i]
    in-arcs from random sources (repeats allowed), the others none."""
    rng = np.random.default_rng(seed)
    dst = np.repeat(np.arange(len(lengths)), lengths)
    src = rng.integers(0, n, dst.shape[0])
    return in_csr_from_edges(n, src.tolist(), dst.tolist(), directed=True)


GRAPHS = {
    # one batch of 8 arcs a lane: each class at its first and last length
    "classes": lambda: graph_of_rows([1, 7, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257] * 9,
                                     700, 1),
    # rows of a whole CTA: up to what one launch takes, and one longer (captured sweeps)
    "hub_rows": lambda: graph_of_rows([2047, 2048, 2049, 9000, 28000, 1, 0, 3], 3000, 2),
    "hubs": lambda: graph_of_rows([2047, 2048, 2049, 9000, 70000, 1, 0, 3], 3000, 2),
    "one_node": lambda: in_csr_from_edges(1, [], [], directed=True),
    "self_loop": lambda: in_csr_from_edges(1, [0], [0], directed=True),
    "two": lambda: in_csr_from_edges(2, [0], [1], directed=True),
    "no_arcs": lambda: in_csr_from_edges(33, [], [], directed=True),
    # more tasks than warps, ragged
    "many_rows": lambda: graph_of_rows([5] * 60001, 200003, 3),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("norm,distribute,normalized", [(0, False, False), (1, True, False),
                                                        (0, True, True)])
def test_small_graphs_match_oracle(oracle_mod, name, norm, distribute, normalized):
    csr = GRAPHS[name]()
    dg = _capi.DeviceGraph(csr)
    p = dg.params(0.85, 1e-10, norm, normalized, distribute, _capi.NKG_PREC_FP64, 5000)
    s, it, mx, st = dg.run(p, trace=64)
    o = oracle_mod.pagerank(csr, tol=1e-10, norm=norm, distribute_sinks=distribute,
                            normalized=normalized, max_iterations=5000)
    scale = max(1.0, float(np.abs(o.scores).sum()))
    assert abs(it - o.iterations) <= 1
    if it == o.iterations:
        assert np.abs(s - o.scores).sum() <= bar(csr.z) * scale
    assert mx == pytest.approx(o.scores.max() if normalized else 1.0, rel=1e-12)
    k = min(it, o.iterations, 64)
    np.testing.assert_allclose(st["residual_trace"][:k], o.trace[:k], rtol=1e-9, atol=bar(csr.z))
    s2, it2, _, _ = dg.run(p)
    np.testing.assert_array_equal(s, s2)
    assert it == it2


def test_small_run_over_several_launches_teleport_and_precisions(oracle_mod):
    csr = GRAPHS["classes"]()
    dg = _capi.DeviceGraph(csr)
    # tol 0: exactly 600 sweeps, three launches of at most 256
    p = dg.params(0.85, 0.0, 0, False, True, _capi.NKG_PREC_FP64, 600)
    s, it, _, _ = dg.run(p)
    o = oracle_mod.pagerank(csr, tol=0.0, norm=0, distribute_sinks=True, max_iterations=600)
    assert it == 600 and np.abs(s - o.scores).sum() <= bar(csr.z)
    t = np.random.default_rng(4).random(csr.z)
    t /= t.sum()
    p = dg.params(0.85, 1e-10, 0, False, True, _capi.NKG_PREC_FP64, 600)
    s, it, _, _ = dg.run(p, t)
    o = oracle_mod.pagerank(csr, tol=1e-10, norm=0, distribute_sinks=True, teleport=t)
    assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-10
    p32 = dg.params(0.85, 1e-7, 0, False, True, _capi.NKG_PREC_FP32, 600)
    s32, _, _, _ = dg.run(p32)
    o = oracle_mod.pagerank(csr, tol=1e-12, norm=0, distribute_sinks=True)
    # 700 FP32 scores of unit mass after a test at 1e-7
    assert np.abs(s32 - o.scores).sum() <= 2e-6


def test_small_run_with_deleted_nodes(oracle_mod):
    gone = (0, 7, 39)
    e = np.random.default_rng(6).integers(0, 40, (300, 2))
    e = e[~np.isin(e, gone).any(axis=1)]
    exists = np.ones(40, np.uint8)
    exists[list(gone)] = 0
    csr = in_csr_from_edges(40, e[:, 0].tolist(), e[:, 1].tolist(), directed=True, exists=exists)
    dg = _capi.DeviceGraph(csr)
    p = dg.params(0.85, 1e-12, 0, False, True, _capi.NKG_PREC_FP64, 5000)
    s, it, _, _ = dg.run(p)
    o = oracle_mod.pagerank(csr, tol=1e-12, norm=0, distribute_sinks=True)
    assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-11


@pytest.mark.parametrize("hub,one_launch", [(28_672, True), (28_900, False), (1_000_000, False)])
def test_a_row_longer_than_a_ctas_share_is_cut_into_chunks(oracle_mod, hub, one_launch):
    """One CTA adds up a row in the one-launch run, so a graph with a longer row
    than 28,672 arcs and half an SM's share takes the captured sweeps."""
    csr = graph_of_rows([hub, 3000, 7, 0, 2], 5000, 11)
    assert 28_672 + csr.arcs // 200 < 28_900 or hub > 100_000  # at least 100 SMs
    dg = _capi.DeviceGraph(csr)
    o = oracle_mod.pagerank(csr, tol=1e-11, norm=0, distribute_sinks=True)
    p = dg.params(0.85, 1e-11, 0, False, True, _capi.NKG_PREC_FP64, 5000)
    s, it, _, st = dg.run(p)
    assert (st["kernel_launches"] == 1) == one_launch
    assert abs(it - o.iterations) <= 1 and np.abs(s - o.scores).sum() <= 1e-11
    p32 = dg.params(0.85, 0.0, 0, False, True, _capi.NKG_PREC_FP32, 60)
    # FP32 scores of unit mass, one of them most of it: a few roundings of 2^-24
    assert np.abs(dg.run(p32)[0] - o.scores).sum() <= 1e-6


@pytest.mark.parametrize("polls,ctas", [(0, 0), (1 << 22, 4096)])
def test_runs_go_on_as_captured_sweeps_where_one_launch_cannot(polls, ctas):
    """A grid barrier that gives up at once, and a grid larger than the GPU holds
    at a time (which the launch refuses): the run is what captured sweeps give."""
    import ctypes as C

    csr = graph_of_rows([300] * 2000, 20_000, 5)
    dg, captured = _capi.DeviceGraph(csr), _capi.DeviceGraph(csr, hot_tier_kb=0)
    f = _capi.lib().nkg_test_small_run
    f.restype, f.argtypes = None, [C.c_void_p, C.c_uint32, C.c_uint32]
    f(dg.h, polls, ctas)
    t = np.random.default_rng(1).random(csr.z)
    for prec, tele in ((_capi.NKG_PREC_FP64, None), (_capi.NKG_PREC_FP32, None),
                       (_capi.NKG_PREC_FP64, t / t.sum())):
        p = dg.params(0.85, 1e-6, 0, False, True, prec, 500)
        s, it, _, st = dg.run(p, tele)
        want, want_it, _, want_st = captured.run(p, tele)
        np.testing.assert_array_equal(s, want)
        assert it == want_it and st["kernel_launches"] == want_st["kernel_launches"] > 1

"""The shared-memory kernel of the many-graph batch against the oracle, at the
edges of its row classes and of the sizes that fit (FP64: 28,536 nodes, FP32:
57,080; larger graphs of the same batch take the other kernel)."""
import numpy as np
import pytest

from networkit_b200 import _capi, generators
from networkit_b200.graph import concat_in_csr, in_csr_from_edges

pytestmark = pytest.mark.gpu


def rows_graph(lengths, n, seed):
    rng = np.random.default_rng(seed)
    dst = np.repeat(np.arange(len(lengths)), lengths)
    src = rng.integers(0, n, dst.shape[0])
    return in_csr_from_edges(n, src.tolist(), dst.tolist(), directed=True)


@pytest.fixture(scope="module")
def batch():
    gs = [rows_graph([1, 7, 8, 9, 31, 32, 33, 64, 65, 128, 129, 255, 256, 257, 4000] * 3, 400, 1),
          in_csr_from_edges(1, [], [], directed=True),
          in_csr_from_edges(3, [0, 1, 2], [1, 2, 0], directed=True),
          generators.hyperbolic(4099, 12, 3, seed=2)]
    # around the FP64 and the FP32 limits of 227 KB - 4 KB
    for i, n in enumerate((28535, 28537, 57079, 57081)):
        gs.append(generators.erdos_renyi(n, 6.0 / n, seed=10 + i))
    csr, offs = concat_in_csr(gs)
    return gs, offs, _capi.DeviceBatch(csr, offs)


@pytest.mark.parametrize("prec", [_capi.NKG_PREC_FP64, _capi.NKG_PREC_FP32])
@pytest.mark.parametrize("norm,distribute,normalized", [(0, False, False), (1, True, False),
                                                        (0, True, True)])
def test_every_graph_matches_oracle(oracle_mod, batch, prec, norm, distribute, normalized):
    gs, offs, db = batch
    fp64 = prec == _capi.NKG_PREC_FP64
    tol = 1e-10 if fp64 else 1e-8
    p = _capi.PRParams(0.85, tol, norm, int(normalized), int(distribute), prec, 10000)
    s, its, floor, st = db.run(p)
    for i, g in enumerate(gs):
        o = oracle_mod.pagerank(g, tol=tol, norm=norm, distribute_sinks=distribute,
                                normalized=normalized)
        scale = max(1.0, float(np.abs(o.scores).sum()))
        err = float(np.abs(s[int(offs[i]):int(offs[i + 1])] - o.scores).sum())
        if fp64:
            assert abs(int(its[i]) - o.iterations) <= 1
            assert err <= 1e-10 * scale, (i, err)
        else:
            # the FP32 rounding floor of a unit-mass vector, and under the L2
            # test the truncation the oracle's own stop leaves
            assert err <= (1e-6 if norm == 0 else 2e-5) * scale, (i, err)
    assert st["kernel_launches"] == 2  # graphs on both sides of the limit
    s2, its2, _, _ = db.run(p)
    np.testing.assert_array_equal(s, s2)
    np.testing.assert_array_equal(its, its2)


def test_iteration_cap_and_graph_times(batch):
    gs, offs, db = batch
    p = _capi.PRParams(0.85, -1.0, 0, 0, 0, _capi.NKG_PREC_FP64, 3)
    _, its, _, st = db.run(p)
    assert (its == 3).all() and st["iterations"] == 3 * len(gs)
    start, end = db.graph_times()
    assert (start >= 0).all() and (end >= start).all()


@pytest.mark.parametrize("prec", [_capi.NKG_PREC_FP64, _capi.NKG_PREC_FP32])
@pytest.mark.parametrize("count", [1, 3, 20])
def test_few_graphs_get_larger_clusters(oracle_mod, count, prec):
    """Up to 16 CTAs a graph, dense ones with hub rows."""
    gs = [rows_graph([9000, 4000, 300] + [70] * (2500 + 37 * i), 3000 + 41 * i, i)
          for i in range(count)]
    csr, offs = concat_in_csr(gs)
    db = _capi.DeviceBatch(csr, offs)
    tol = 1e-10 if prec == _capi.NKG_PREC_FP64 else 1e-8
    s, its, _, st = db.run(_capi.PRParams(0.85, tol, 0, 0, 1, prec, 10000))
    assert st["kernel_launches"] == 1
    for i, g in enumerate(gs):
        o = oracle_mod.pagerank(g, tol=tol, norm=0, distribute_sinks=True)
        err = float(np.abs(s[int(offs[i]):int(offs[i + 1])] - o.scores).sum())
        assert err <= (1e-10 if prec == _capi.NKG_PREC_FP64 else 1e-6), (i, err)

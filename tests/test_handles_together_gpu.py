"""Handles of different sizes used in turn and on two threads: a call's launch
limits must not depend on what another handle of the process ran before it."""
import threading

import numpy as np
import pytest

from networkit_b200 import _capi, generators
from networkit_b200.graph import concat_in_csr

pytestmark = pytest.mark.gpu

F64, F32 = _capi.NKG_PREC_FP64, _capi.NKG_PREC_FP32


def er_batch(n, count):
    return _capi.DeviceBatch(*concat_in_csr(
        [generators.erdos_renyi(n, 8.0 / n, seed=i) for i in range(count)]))


@pytest.mark.parametrize("prec", [F64, F32])
def test_batch_runs_again_after_a_batch_of_smaller_graphs(prec):
    p = _capi.PRParams(0.85, 1e-8, 0, 0, 0, prec, 1000)
    large, small = er_batch(28000, 2), er_batch(1000, 2)
    want = large.run(p)[0]
    small.run(p)
    for shape in ((8, 512, 64), (2, 256, 128)):  # each captures the launch anew
        large.set_tuning(*shape)
        np.testing.assert_array_equal(large.run(p)[0], want)


def test_tier_graph_runs_again_after_a_smaller_tier():
    csr = generators.rmat_directed(16, 16, seed=2)
    large, small = (_capi.DeviceGraph(csr, hot_tier_kb=kb) for kb in (200, 144))
    for prec in (F64, _capi.NKG_PREC_FP32_REFINE):
        p = large.params(0.85, 1e-10, 0, False, True, prec, 1000)
        want = large.run(p)[0]
        small.run(p)
        t = np.zeros(csr.z)
        t[3] = 1.0
        # a teleport run captures its sweeps anew; a refinement launches them
        np.testing.assert_array_equal(large.run(p)[0], want)
        assert np.abs(large.run(p, t)[0] - small.run(p, t)[0]).sum() <= 2e-9


def on_two_threads(calls):
    """Each call on a thread of its own, at the same time; their errors."""
    errors = []

    def work(call):
        try:
            call()
        except BaseException as e:  # handed to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_wide_ppr_on_two_threads():
    csr = generators.rmat_directed(12, 16, seed=5)
    ks = (256, 130)
    handles = [_capi.DeviceGraph(csr) for _ in ks]
    seeds = [np.arange(k, dtype=np.uint32) for k in ks]
    p = handles[0].params(0.85, 1e-7, 0, False, True, F32, 100)
    want = [h.ppr(s, p)[0] for h, s in zip(handles, seeds)]

    def again(i):
        for _ in range(40):
            np.testing.assert_array_equal(handles[i].ppr(seeds[i], p)[0], want[i])

    on_two_threads([lambda: again(0), lambda: again(1)])


def test_one_launch_runs_and_batches_on_two_threads():
    """Whole-GPU launches (a grid barrier, clusters) of different streams."""
    g = _capi.DeviceGraph(generators.rmat_directed(17, 16, seed=6))
    b = er_batch(20000, 4)
    g2 = _capi.DeviceGraph(generators.rmat_directed(16, 16, seed=7))
    pg = g.params(0.85, 1e-9, 0, False, True, F64, 500)
    pb = _capi.PRParams(0.85, 1e-8, 0, 0, 0, F32, 1000)
    want, launches = g.run(pg)[0], g.run(pg)[3]["kernel_launches"]
    want2, want_b = g2.run(pg)[0], b.run(pb)[0]
    assert launches == 1

    def graph(h, w):
        for _ in range(60):
            np.testing.assert_array_equal(h.run(pg)[0], w)

    def batch():
        for _ in range(60):
            np.testing.assert_array_equal(b.run(pb)[0], want_b)

    on_two_threads([lambda: graph(g, want), lambda: graph(g2, want2)])
    on_two_threads([lambda: graph(g, want), batch])

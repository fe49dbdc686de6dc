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


def test_wide_ppr_on_two_threads():
    csr = generators.rmat_directed(12, 16, seed=5)
    ks = (256, 130)  # 192 and 215 KB of shared memory
    handles = [_capi.DeviceGraph(csr) for _ in ks]
    seeds = [np.arange(k, dtype=np.uint32) for k in ks]
    p = handles[0].params(0.85, 1e-7, 0, False, True, F32, 100)
    want = [h.ppr(s, p)[0] for h, s in zip(handles, seeds)]
    errors = []

    def work(i):
        try:
            for _ in range(40):
                np.testing.assert_array_equal(handles[i].ppr(seeds[i], p)[0], want[i])
        except BaseException as e:  # handed to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors

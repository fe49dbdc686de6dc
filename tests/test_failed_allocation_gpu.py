"""A call that runs out of device memory leaves its handle usable: made again,
it gives what an untroubled handle gives. Every device allocation of the call
fails in turn."""
import numpy as np
import pytest

from networkit_b200 import _capi, generators
from networkit_b200.graph import concat_in_csr

pytestmark = pytest.mark.gpu

F64, F32, REFINE = _capi.NKG_PREC_FP64, _capi.NKG_PREC_FP32, _capi.NKG_PREC_FP32_REFINE


@pytest.fixture(scope="module")
def csr():
    csr = generators.rmat_directed(12, 16, seed=5)
    assert int(np.diff(csr.in_ptr).max()) > 256  # rows of several chunks
    return csr


def graph(csr, **kw):
    return _capi.DeviceGraph(csr, **kw)


def ppr(g, k):
    p = g.params(0.85, 1e-7, 0, False, True, F32, 100)
    return g.ppr(np.arange(k, dtype=np.uint32), p)[0]


def run(g, prec):
    return g.run(g.params(0.85, 1e-9, 0, False, True, prec, 500))[0]


def new_weights(g):
    g.set_weights(np.linspace(0.5, 1.0, int(g.info()["arcs"])))
    return run(g, F64)


def batch():
    gs = [generators.rmat_directed(10, 8, seed=3), generators.erdos_renyi(30000, 2e-4, seed=4),
          generators.erdos_renyi(60000, 1e-4, seed=5)]
    return _capi.DeviceBatch(*concat_in_csr(gs))


CALLS = {
    "ppr_narrow": (graph, lambda g: ppr(g, 9)),
    "ppr_wide": (graph, lambda g: ppr(g, 130)),
    "small_run": (graph, lambda g: run(g, F64)),
    "captured_fp64": (lambda c: graph(c, hot_tier_kb=0), lambda g: run(g, F64)),
    "captured_fp32": (lambda c: graph(c, sweep_shape=1), lambda g: run(g, F32)),
    "refine": (graph, lambda g: run(g, REFINE)),
    "set_weights": (lambda c: graph(generators.with_uniform_weights(c, seed=1)), new_weights),
    "batch_fp32": (lambda c: batch(), lambda b: b.run(_capi.PRParams(0.85, 1e-8, 0, 0, 0, F32,
                                                                     500))[0]),
    "batch_fp64": (lambda c: batch(), lambda b: b.run(_capi.PRParams(0.85, 1e-8, 0, 0, 0, F64,
                                                                     500))[0]),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_a_call_is_whole_again_after_a_failed_allocation(fail_alloc, csr, name):
    make, call = CALLS[name]
    want = call(make(csr))
    failures = 0
    for k in range(200):
        h = make(csr)
        fail_alloc(k)
        try:
            got = call(h)
        except _capi.NkgError as e:
            assert e.code == _capi.NKG_ERR_OOM
            failures += 1
            got = call(h)
        else:
            assert fail_alloc(-1) >= 0  # fewer than k + 1 allocations
            np.testing.assert_array_equal(got, want)
            break
        np.testing.assert_array_equal(got, want)
    assert 0 < failures < 200

"""The many-graph batch's kernel for larger graphs at every launch shape and
variant, on graphs of every kind (which the library itself gives to the
shared-memory kernel), and what the tuning does where no graph uses it."""
import ctypes as C

import numpy as np
import pytest

from networkit_b200 import _capi, generators
from networkit_b200.graph import concat_in_csr
from test_batch_gpu import DAMP, check, mixed_graphs

pytestmark = pytest.mark.gpu

F64, F32 = _capi.NKG_PREC_FP64, _capi.NKG_PREC_FP32


def shared_up_to(db, nodes):
    f = _capi.lib().nkg_test_batch_shared
    f.restype, f.argtypes = None, [C.c_void_p, C.c_uint32]
    f(db.h, nodes)
    return db


@pytest.fixture(scope="module", params=[0, 2000])
def batch(request):
    """Every graph in the larger graphs' kernel, and half of them."""
    gs = mixed_graphs()
    csr, offs = concat_in_csr(gs)
    return gs, offs, shared_up_to(_capi.DeviceBatch(csr, offs), request.param), request.param


@pytest.mark.parametrize("shape", [(1, 128, 4, 0), (2, 256, 32, 1), (4, 512, 128, 2),
                                   (8, 256, 1024, 3), (16, 256, 64, 0)])
@pytest.mark.parametrize("prec", [F64, F32])
def test_every_shape_matches_oracle(oracle_mod, batch, shape, prec):
    gs, offs, db, nodes = batch
    db.set_tuning(*shape)
    tol = 1e-10 if prec == F64 else 1e-8
    p = _capi.PRParams(DAMP, tol, 0, 0, 0, prec, 10000)
    s, its, _, st = db.run(p)
    check(oracle_mod, gs, offs, s, its, prec, 0, tol, False, False)
    assert st["kernel_launches"] == (2 if nodes else 1)
    s2, its2, _, _ = db.run(p)
    np.testing.assert_array_equal(s, s2)
    np.testing.assert_array_equal(its, its2)


@pytest.mark.parametrize("norm,distribute,normalized", [(1, False, False), (0, True, False),
                                                        (0, False, True)])
def test_options_match_oracle(oracle_mod, batch, norm, distribute, normalized):
    gs, offs, db, _ = batch
    db.set_tuning(4, 256, 64)
    p = _capi.PRParams(DAMP, 1e-9, norm, int(normalized), int(distribute), F64, 10000)
    s, its, _, _ = db.run(p)
    check(oracle_mod, gs, offs, s, its, F64, norm, 1e-9, distribute, normalized)


def test_tuning_without_larger_graphs_is_kept():
    csr, offs = concat_in_csr([generators.erdos_renyi(2000, 4e-3, seed=i) for i in range(4)])
    db = _capi.DeviceBatch(csr, offs)
    db.set_tuning(2, 512, 64)
    p = _capi.PRParams(DAMP, 1e-8, 0, 0, 0, F32, 100)
    best, table = db.tune(p, sweeps=4)
    assert len({t["ms"] for t in table}) == 1  # one run stands for all
    for t in (best, db.tuning()):
        assert (t["cluster"], t["threads"], t["split"]) == (2, 512, 64)


def test_tuning_with_larger_graphs_times_every_shape():
    db = shared_up_to(_capi.DeviceBatch(*concat_in_csr(
        [generators.erdos_renyi(2000, 4e-3, seed=i) for i in range(4)])), 0)
    best, table = db.tune(_capi.PRParams(DAMP, 1e-8, 0, 0, 0, F32, 100), sweeps=20)
    assert len(table) > 20 and len({t["ms"] for t in table}) > 10
    assert best["ms"] == min(t["ms"] for t in table)
    assert {t["variant"] for t in table} == {0, 1, 2, 3}

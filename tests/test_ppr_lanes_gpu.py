"""Personalised PageRank columns for every way a row's columns are laid over
the lanes of a warp: one to 32 lanes, several groups of lanes on different arcs (up to 64
columns), one arc per warp with 4 or 8 columns a lane (more)."""
import numpy as np
import pytest

from networkit_b200 import _capi, generators

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    csr = generators.rmat_directed(13, 16, seed=9)  # sinks, rows of several chunks
    dg = _capi.DeviceGraph(csr)
    assert int(np.diff(csr.in_ptr).max()) > 600
    return csr, dg


@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 17, 31, 37, 56, 63, 64, 65, 72, 100, 127, 128, 129,
                               137, 200, 255, 256])
def test_columns_match_the_fp64_run(graph, k):
    csr, dg = graph
    seeds = np.random.default_rng(k).choice(csr.z, k, replace=False).astype(np.uint32)
    p = dg.params(0.85, 1e-7, 0, False, True, _capi.NKG_PREC_FP32, 300)
    s, its, _ = dg.ppr(seeds, p)
    assert s.shape == (k, csr.z) and (its > 1).all()
    s2, its2, _ = dg.ppr(seeds, p)
    np.testing.assert_array_equal(s, s2)
    np.testing.assert_array_equal(its, its2)
    p64 = dg.params(0.85, 1e-12, 0, False, True, _capi.NKG_PREC_FP64, 2000)
    for j in sorted({0, k // 2, k - 1}):
        t = np.zeros(csr.z)
        t[seeds[j]] = 1.0
        # FP32 bar of the companion forms; columns sum to 1
        assert np.abs(s[j] - dg.run(p64, t)[0]).sum() <= 1e-6, j

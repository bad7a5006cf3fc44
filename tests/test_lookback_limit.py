"""The look-back waits of the scans and sorts, made to run out by a limit that
any wait exceeds: a call then ends with TDT_ERR_TIMEOUT, whatever indexes by a
sort or scan that gave up stays inside its arrays, and the next call is exact."""
import numpy as np
import pytest
import torch

from tdtdecomposition_gb300 import _lib, generators as G, truss as T
from tdtdecomposition_gb300.preprocess import _check_status, preprocess_edges


def test_status_messages():
    _check_status(0)
    with pytest.raises(_lib.TdtError, match="vertex id outside") as e:
        _check_status(_lib.ERR_INVALID)
    assert e.value.status == 1
    with pytest.raises(_lib.TdtError, match="timed out") as e:
        _check_status(_lib.ERR_TIMEOUT)
    assert "vertex id" not in str(e.value) and e.value.status == 4


def _calls_that_time_out(call, exact, calls=30):
    """Of `calls` calls under the limit, those that ran out; the others are exact."""
    n = 0
    _lib.load().tdt_set_lookback_limit_ns(1)
    try:
        for _ in range(calls):
            try:
                exact(call())
            except _lib.TdtError as e:
                assert e.status == _lib.ERR_TIMEOUT
                n += 1
    finally:
        _lib.load().tdt_set_lookback_limit_ns(0)
    exact(call())
    return n


@pytest.mark.gpu
@pytest.mark.parametrize("m", [5000, 300001, 2000003])
def test_preprocess_waits_run_out(m):
    rng = np.random.default_rng(m)
    s, d = (torch.as_tensor(rng.integers(0, m // 8, m).astype(np.int32)).cuda() for _ in range(2))
    g0, v0 = preprocess_edges(s, d)

    def exact(r):
        g, v = r
        assert torch.equal(g.columns, g0.columns) and torch.equal(g.row_ptr, g0.row_ptr) and torch.equal(v, v0)

    n = _calls_that_time_out(lambda: preprocess_edges(s, d), exact)
    assert n > 0 or m < 100000  # some hundred tiles start at once


@pytest.mark.gpu
@pytest.mark.parametrize("route", [0, 1, 2])
def test_decompose_waits_run_out(route):
    g, _ = preprocess_edges(*G.rmat_edges_device(16, 16 << 16, seed=2))
    t = T.triangle_count(g)
    budget = {0: 0, 1: 24 * t + 256, 2: 24 * t + T.stage_bytes(g.columns, g.row_ptr) + 256}[route]
    want = T.truss_decompose(g, list_budget=budget)
    assert want.listing == route

    def exact(r):
        assert torch.equal(r.truss, want.truss) and torch.equal(r.e_truss, want.e_truss)

    assert _calls_that_time_out(lambda: T.truss_decompose(g, list_budget=budget), exact) > 0

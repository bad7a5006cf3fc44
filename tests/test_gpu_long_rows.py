"""Validation of rows that are derived, where a block takes over a long one:
rows at the bound, more long rows than a block keeps, faults at the ends and
inside of a long row, and a hub whose check does not grow into a chain."""
import numpy as np
import pytest
import torch

from tdtdecomposition_gb300 import CSRCOO, _lib, truss as T

pytestmark = pytest.mark.gpu
LONG = 2048


def _stars(lengths):
    """Row i of lengths[i] edges to the ids that follow the rows."""
    n = len(lengths)
    cols = np.concatenate([n + np.arange(k) for k in lengths]).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(lengths), np.full(max(lengths), sum(lengths))]).astype(np.int64)
    return cols, rp


def _count(cols, rp):
    g = CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).cuda())
    return T.triangle_count(g)


@pytest.mark.parametrize("lengths", [[LONG], [LONG + 1], [LONG - 1, LONG + 1, 1, 3 * LONG + 5], [LONG + 1] * 40000])
def test_long_rows_are_accepted(lengths):
    cols, rp = _stars(lengths)
    assert _count(cols, rp) == 0
    r = T.truss_decompose(CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).cuda()), lists=False)
    assert r.kmax == 2


@pytest.mark.parametrize("at", [1, 255, 256, 1023, 1024, LONG - 1, LONG, 5 * LONG])
def test_faults_in_long_rows(at):
    cols, rp = _stars([5, 5 * LONG + 1, 7])
    for bad in (cols[5 + at - 1], -1, len(rp)):  # not increasing, negative, past the vertices
        c = cols.copy()
        c[5 + at] = bad
        with pytest.raises(_lib.TdtError):
            _count(c, rp)


def test_a_hub_is_checked_in_time():
    """One row of 2 M edges; derived by one warp, load after load, 39 ms."""
    cols, rp = _stars([2000000])
    g = CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).cuda())
    ms = []
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        assert T.triangle_count(g) == 0
        b.record()
        torch.cuda.synchronize()
        ms.append(a.elapsed_time(b))
    assert min(ms) < 6.0

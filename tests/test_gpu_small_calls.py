"""Validation without given rows (a warp per row writes and checks them), the
triangle count that ends with its last block, and the stats words of a call
that failed: rows at the 32-lane edges, malformed row pointers and columns."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import CSRCOO, _lib, truss as T

pytestmark = pytest.mark.gpu


def _graph(rp, cols, rows=None):
    t = lambda a, d: torch.as_tensor(np.asarray(a, d)).cuda()
    return CSRCOO(columns=t(cols, np.int32), row_ptr=t(rp, np.int64), rows=None if rows is None else t(rows, np.int32))


def _clique(n):
    r, c = np.triu_indices(n, 1)
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c, r


@pytest.mark.parametrize("n", [2, 3, 32, 33, 34, 65, 257])
def test_rows_derived_or_given(n):
    rp, c, r = _clique(n)
    for rows in (None, r):
        tri, sup = T.triangle_count(_graph(rp, c, rows), return_support=True)
        assert tri == n * (n - 1) * (n - 2) // 6
        assert (sup.cpu().numpy() == n - 2).all()
        assert T.triangle_count(_graph(rp, c, rows)) == tri
        assert T.truss_decompose(_graph(rp, c, rows)).kmax == n
        assert bool(T.ktruss_search(_graph(rp, c, rows), n).all())


def _broken():
    rp, c, r = _clique(40)
    bad = c.copy()
    bad[[5, 6]] = bad[[6, 5]]
    yield "unsorted", rp, bad
    bad = c.copy()
    bad[39] = 1  # row 1 points at itself
    yield "self", rp, bad
    bad = c.copy()
    bad[7] = 40
    yield "column range", rp, bad
    bad = c.copy()
    bad[7] = -1
    yield "negative column", rp, bad
    bad = rp.copy()
    bad[3] = bad[4] + 1
    yield "falling row pointer", bad, c
    bad = rp.copy()
    bad[-1] += 1
    yield "end", bad, c
    bad = rp.copy()
    bad[0] = 1
    yield "begin", bad, c


@pytest.mark.parametrize("name,rp,c", list(_broken()), ids=[b[0] for b in _broken()])
def test_malformed_is_refused(name, rp, c):
    g = _graph(rp, c)
    for call in (lambda: T.triangle_count(g), lambda: T.truss_decompose(g, lists=False),
                 lambda: T.truss_decompose(g, list_budget=1 << 20)):
        with pytest.raises(_lib.TdtError):
            call()
    stats = T.truss_decompose(g, lists=False, sync=False)[3].cpu()
    assert int(stats[T.STAT_STATUS]) != 0 and int(stats[1:].abs().sum()) == 0


@pytest.mark.parametrize("n", [1, 31, 32, 255, 256, 257, 100003, 3000001])
def test_max_id(n):
    from tdtdecomposition_gb300.preprocess import _max_id
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, 1 << 31, n, dtype=np.int64).astype(np.int32), rng.integers(0, 1 << 30, n + 5).astype(np.int32)
    a[rng.integers(n)] = (1 << 31) - 1 if n % 2 else 7
    ca, cb = torch.as_tensor(a).cuda(), torch.as_tensor(b).cuda()
    assert _max_id(ca, cb) == max(int(a.max()), int(b.max()))
    assert _max_id(ca[n - 1:]) == int(a[-1])
    with pytest.raises(RuntimeError):
        _max_id(ca, ca[:0])

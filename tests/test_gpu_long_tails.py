"""Orders that are not degree ranks: sources of many out-edges that rank low,
whose tails are far longer than the rows they meet in the walk.  Results against
the oracle by every route, and a walk that is linear in the edges."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import CSRCOO, _lib, truss as T

pytestmark = pytest.mark.gpu


def _graph(pairs, V):
    lo, hi = pairs.min(1).astype(np.int64), pairs.max(1).astype(np.int64)
    k = np.unique(lo[lo != hi] * V + hi[lo != hi])
    rows, cols = (k // V).astype(np.int32), (k % V).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=V))])
    return rows, cols, rp


def _wheel(n):
    """Hub 0 joined to the n - 1 vertices of a ring."""
    i = np.arange(1, n)
    return np.concatenate([np.stack([np.zeros_like(i), i], 1), np.stack([i, np.where(i + 1 < n, i + 1, 1)], 1)])


def _hubs(n, hubs, m, seed):
    """Low hubs joined to each other and to all of n vertices with m random edges."""
    rng = np.random.default_rng(seed)
    h, i = np.arange(hubs), np.arange(hubs, hubs + n)
    a, b = np.triu_indices(hubs, 1)
    return np.concatenate([np.stack([a, b], 1), np.stack([np.repeat(h, n), np.tile(i, hubs)], 1),
                           rng.integers(hubs, hubs + n, (m, 2))])


def _tail(n, d):
    """Source 0 of n out-edges; source 1, its first, of the last d of them: a row
    of d entries behind a tail of n - 1."""
    i = np.arange(1, n + 1)
    return np.concatenate([np.stack([np.zeros_like(i), i], 1), np.stack([np.ones(d, np.int64), i[n - d:]], 1)])


def _bipartite(n):
    """n x n joined, and a path through the second half: block rows of one entry."""
    a, b = np.meshgrid(np.arange(n), n + np.arange(n))
    i = n + np.arange(n - 1)
    return np.concatenate([np.stack([a.ravel(), b.ravel()], 1), np.stack([i, i + 1], 1)])


GRAPHS = {
    "wheel": (lambda: _wheel(12000), 12000),
    "hubs": (lambda: _hubs(6000, 40, 30000, 1), 6040),       # several runs a warp, rows of all kinds
    "hubs_dense": (lambda: _hubs(9000, 3, 400000, 2), 9003),  # block rows with long tails
    "tail_128": (lambda: _tail(129, 2), 130),                 # the longest tail that is streamed
    "tail_129": (lambda: _tail(130, 2), 131),
    "ratio_at": (lambda: _tail(4 * 80 + 1, 80), 4 * 80 + 2),
    "ratio_past": (lambda: _tail(4 * 80 + 2, 80), 4 * 80 + 3),
    "warp_row": (lambda: _tail(4 * 256 + 2, 256), 4 * 256 + 3),
    "block_row": (lambda: _tail(4 * 257 + 2, 257), 4 * 257 + 3),
    "chunked_row": (lambda: _tail(4 * 5000 + 2, 5000), 4 * 5000 + 3),
    "bipartite": (lambda: _bipartite(300), 600),
}


@pytest.mark.parametrize("caps", [(0, 0), (3, 16)])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_long_tails_vs_oracle(name, caps):
    make, V = GRAPHS[name]
    rows, cols, rp = _graph(make(), V)
    sup_ref = O.support(rows, cols, rp.astype(np.int32), 1)
    kmax, et, pt, truss = O.k_truss(rows, cols, O.tiling_row_ptr(rows, cols, V, 1), V, 1)
    g = CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).cuda(), rows=torch.as_tensor(rows).cuda())
    _lib.load().tdt_set_support_caps(*caps)
    try:
        t, sup = T.triangle_count(g, return_support=True)
        assert t == int(sup_ref.sum()) // 3 and np.array_equal(sup.cpu().numpy(), sup_ref)
        stage = T.stage_bytes(g.columns, g.row_ptr)
        for route, budget in ((0, 0), (1, 24 * t + 256), (2, 24 * t + stage + 256)):
            if budget > 1 << 33:
                continue
            r = T.truss_decompose(g, list_budget=budget)
            assert r.listing == route and r.kmax == kmax
            assert np.array_equal(r.truss.cpu().numpy(), truss) and np.array_equal(r.e_truss.cpu().numpy(), et)
        k = max(3, kmax - 1)
        assert np.array_equal(T.ktruss_search(g, k, lists=False).cpu().numpy(), truss >= k)
    finally:
        _lib.load().tdt_set_support_caps(0, 0)


def test_low_hub_is_linear():
    """A wheel of 200,000 vertices: the walk from the source took 2.0 to 2.4 ms
    of support phase, whole tails 28 ms."""
    n = 200000
    rows, cols, rp = _graph(_wheel(n), n)
    g = CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).cuda(), rows=torch.as_tensor(rows).cuda())
    ms = []
    for _ in range(5):
        with T.PhaseProfile() as p:
            r = T.truss_decompose(g, lists=False)
        ms.append(p.ms["support"])
    assert r.kmax == 3 and r.triangles == n - 1
    assert min(ms) < 5.0

"""The search peel with a compacted adjacency: rows a warp and rows a block
compacts (an in-list past a thousand entries), compactions that leave items
queued before them, and a list tail too small for the lists (the search kernel
then follows the listed one); against the listed peel and the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import CSRCOO, _lib, generators as G, truss as T
from tdtdecomposition_gb300.preprocess import preprocess_edges

pytestmark = pytest.mark.gpu


def _hub(n, m, seed):
    """Two hubs joined to n vertices among which m random edges run: in-lists
    of n entries that shrink level by level."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    return np.concatenate([np.stack([i, np.full(n, n)], 1), np.stack([i, np.full(n, n + 1)], 1), [[n, n + 1]],
                           rng.integers(0, n, (m, 2))]).astype(np.int32)


GRAPHS = {
    "hub_1024": lambda: _hub(1024, 30000, 1),     # the block row bound and one past it
    "hub_1025": lambda: _hub(1025, 30000, 2),
    "hub_5000": lambda: _hub(5000, 60000, 3),     # several tiles of a block row, the last one ragged
    "chung_lu": lambda: np.stack(G.chung_lu_edges(30000, seed=4), 1),
    "tiny": lambda: np.array([[0, 1], [1, 2], [0, 2], [2, 3]], np.int32),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_compacted_search_vs_oracle(name):
    rows, cols, rp, verts = O.preprocess(GRAPHS[name](), stable=True)
    V = len(verts)
    kmax, et, pt, truss = O.k_truss(rows, cols, O.tiling_row_ptr(rows, cols, V, 1), V, 1)
    g = CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).long().cuda(),
               rows=torch.as_tensor(rows).cuda())
    for half_sms in (0, 1):
        _lib.load().tdt_set_peel_grid(half_sms)
        try:
            r = T.truss_decompose(g, lists=False)
        finally:
            _lib.load().tdt_set_peel_grid(0)
        assert not r.listed and r.kmax == kmax
        assert np.array_equal(r.truss.cpu().numpy(), truss) and np.array_equal(r.e_truss.cpu().numpy(), et)
        assert np.array_equal(r.ptr_truss.cpu().numpy(), pt)


def test_lists_that_do_not_fit_a_large_graph():
    """Past 2^20 edges a tail without room for the lists leaves the peel to the
    search kernel that follows."""
    s, d = G.rmat_edges_device(17, 16 << 17, seed=3)
    g, _ = preprocess_edges(s, d)
    assert g.num_edges > 1 << 20
    a = T.truss_decompose(g, lists=True)
    b = T.truss_decompose(g, list_budget=4096)
    c = T.truss_decompose(g, lists=False)
    assert a.listed and not b.listed and not c.listed
    for r in (b, c):
        assert r.kmax == a.kmax and r.rounds == a.rounds
        assert torch.equal(r.truss, a.truss) and torch.equal(r.e_truss, a.e_truss)

"""The middle-vertex walk and its lists where its paths change: rows with more
in-edges than one unit takes, rows wider than the warp's and the block's
bitmaps, columns that start off a 16-byte boundary, and lists taken from the
staging slots or from a second walk; against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import CSRCOO, truss as T

pytestmark = pytest.mark.gpu


def _hubs(n, hubs):
    """`hubs` vertices joined to each other and to all of n others, which form
    a sparse ring: middle vertices with n in-edges and a few out-edges."""
    h = np.arange(n, n + hubs)
    a, b = np.triu_indices(hubs, 1)
    e = [np.stack([h[a], h[b]], 1), np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)]
    e += [np.stack([np.arange(n), np.full(n, x)], 1) for x in h]
    return np.concatenate(e).astype(np.int32)


def _random(n, m, seed):
    return np.random.default_rng(seed).integers(0, n, (m, 2)).astype(np.int32)


GRAPHS = {
    "parts": lambda: _hubs(33001, 4),             # 3 units of 16,384 in-edges, the last one short
    "one_part": lambda: _hubs(16384, 2),          # exactly one full unit
    "parts_dense": lambda: np.concatenate([_hubs(20001, 60), _random(20000, 100000, 4)]),  # a hub's runs, sorted
    "light_wide": lambda: _random(150001, 600000, 1),    # warp rows past 2^13 ids
    "block_wide": lambda: _random(140001, 4200000, 2),   # block rows past 2^16 ids
    "dense": lambda: _random(700, 150000, 3),     # rows of more than 256 out-edges
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_walk_paths_vs_oracle(name, shift):
    rows, cols, rp, verts = O.preprocess(GRAPHS[name](), stable=True)
    sup_ref = O.support(rows, cols, rp.astype(np.int32), 1)
    buf = torch.zeros(len(cols) + shift, dtype=torch.int32, device="cuda")
    buf[shift:] = torch.as_tensor(cols).cuda()
    g = CSRCOO(columns=buf[shift:], row_ptr=torch.as_tensor(rp).long().cuda(), rows=torch.as_tensor(rows).cuda())
    t, sup = T.triangle_count(g, return_support=True)
    assert t == int(sup_ref.sum()) // 3 and np.array_equal(sup.cpu().numpy(), sup_ref)
    stage = T.stage_bytes(g.columns, g.row_ptr)
    search = T.truss_decompose(g, lists=False)
    for route, budget in ((2, 24 * t + stage + 256), (1, 24 * t + 256)):
        r = T.truss_decompose(g, list_budget=budget)
        assert r.listing == route
        assert r.kmax == search.kmax and torch.equal(r.truss, search.truss) and torch.equal(r.e_truss, search.e_truss)
    if shift == 0:
        V = len(verts)
        kmax, et, pt, tr = O.k_truss(rows, cols, O.tiling_row_ptr(rows, cols, V, 1), V, 1)
        assert search.kmax == kmax and np.array_equal(search.truss.cpu().numpy(), tr)
        assert np.array_equal(search.e_truss.cpu().numpy(), et)

"""The short listed sub-rounds at their window edges: disjoint cliques and
books whose sub-rounds hold 31 / 32 / 33 slots, whole warps' windows, items of
one slot and items longer than a window, against the search peel (no slot
index) and the oracle; on the smallest grid, so that sub-rounds pass from the
short path to the long one and back."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import CSRCOO, _lib, generators as G, truss as T

pytestmark = pytest.mark.gpu


def _cliques(sizes):
    out, base = [], 0
    for k in sizes:
        a, b = np.triu_indices(k, 1)
        out.append(np.stack([a + base, b + base], 1))
        base += k
    return np.concatenate(out).astype(np.int32)


GRAPHS = {
    "one_slot": lambda: _cliques([3]),
    "ones": lambda: _cliques([3] * 11 + [4] * 5),             # 33 one-slot items in a round
    "window": lambda: _cliques([3] * 32 + [34, 66]),          # 96 slots; items of 32 and of 64 slots
    "long": lambda: _cliques([3, 5, 130, 258]),               # items of 128 and 256 slots, 33 K of them
    "rmat": lambda: np.stack(G.rmat_edges(15, 12 << 15, seed=9), 1),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("half_sms", [0, 1, 4])
def test_lean_rounds_vs_oracle(name, half_sms):
    rows, cols, rp, verts = O.preprocess(GRAPHS[name](), stable=True)
    V = len(verts)
    kmax, et, pt, truss = O.k_truss(rows, cols, O.tiling_row_ptr(rows, cols, V, 1), V, 1)
    g = CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).long().cuda(),
               rows=torch.as_tensor(rows).cuda())
    L = _lib.load()
    L.tdt_set_peel_grid(half_sms)
    try:
        for lists in (True, False):
            r = T.truss_decompose(g, lists=lists)
            assert r.listed == lists and r.kmax == kmax
            assert np.array_equal(r.truss.cpu().numpy(), truss) and np.array_equal(r.e_truss.cpu().numpy(), et)
        for k in (3, max(3, kmax // 2), kmax):
            m = T.ktruss_search(g, k, lists=True)
            assert np.array_equal(m.cpu().numpy(), truss >= k)
    finally:
        L.tdt_set_peel_grid(0)

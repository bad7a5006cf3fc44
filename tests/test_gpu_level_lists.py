"""Level changes that keep the alive list, rewrite it, or need a second pass
over either: disjoint cliques, whose edges' truss numbers are their sizes, with
levels that kill few edges, most of them, and levels far apart."""
import numpy as np
import pytest
import torch

from tdtdecomposition_gb300 import CSRCOO, truss as T

pytestmark = pytest.mark.gpu


def _cliques(sizes):
    r, c, k, at = [], [], [], 0
    for n in sizes:
        a, b = np.triu_indices(n, 1)
        r.append(a + at)
        c.append(b + at)
        k.append(np.full(len(a), n))
        at += n
    r, c, k = np.concatenate(r), np.concatenate(c), np.concatenate(k)
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=at))])
    g = CSRCOO(columns=torch.as_tensor(c.astype(np.int32)).cuda(), row_ptr=torch.as_tensor(rp).cuda())
    return g, k


@pytest.mark.parametrize("lists", [True, False])
@pytest.mark.parametrize("sizes", [list(range(3, 41)), [40] * 30 + [3, 4, 5], [3] * 4000 + [4, 9, 30, 60], [2, 2, 3],
                                   [120] + list(range(3, 30, 4)), [4] * 9000 + [5] * 700 + [6] * 500])
def test_levels_of_cliques(sizes, lists):
    g, k = _cliques(sizes)
    for _ in range(2):
        r = T.truss_decompose(g, lists=lists)
        assert np.array_equal(r.truss.cpu().numpy(), k)
        assert r.kmax == max(sizes)
        assert r.rounds == len(set(sizes))

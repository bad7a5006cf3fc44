"""Preprocessing and the peel order at the tile edges of the look-back scan,
sort and unique passes: draws and edges of one key less, exactly and one more
than a tile, heavy repetition, one hub, id gaps longer than a warp fills, and
groups; against numpy."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import CSRCOO, truss as T
from tdtdecomposition_gb300.preprocess import preprocess_edges

pytestmark = pytest.mark.gpu


def _numpy_preprocess(s, d, group=None):
    keep = s != d
    lo, hi = np.minimum(s, d)[keep].astype(np.int64), np.maximum(s, d)[keep].astype(np.int64)
    u = np.unique(np.stack([lo, hi], 1), axis=0)
    n = int(max(s.max(), d.max())) + 1
    deg = np.bincount(u.ravel(), minlength=n)
    ids = np.where(deg > 0)[0]
    g = np.zeros(n, np.int64) if group is None else group[:n].astype(np.int64)
    verts = ids[np.lexsort((ids, deg[ids], g[ids]))]
    rank = np.full(n, -1, np.int64)
    rank[verts] = np.arange(len(verts))
    a, b = rank[u[:, 0]], rank[u[:, 1]]
    r, c = np.minimum(a, b), np.maximum(a, b)
    o = np.lexsort((c, r))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=len(verts)))])
    return r[o], c[o], rp, verts


def _check(s, d, group=None):
    s, d = np.asarray(s, np.int32), np.asarray(d, np.int32)
    g, v = preprocess_edges(torch.as_tensor(s).cuda(), torch.as_tensor(d).cuda(),
                            None if group is None else torch.as_tensor(group.astype(np.int32)).cuda())
    r, c, rp, verts = _numpy_preprocess(s, d, group)
    assert np.array_equal(g.rows.cpu().numpy(), r) and np.array_equal(g.columns.cpu().numpy(), c)
    assert np.array_equal(g.row_ptr.cpu().numpy(), rp) and np.array_equal(v.cpu().numpy(), verts)


@pytest.mark.parametrize("m", [1, 31, 2047, 2048, 2049, 3071, 3072, 3073, 4096, 3 * 3072 + 5, 700001])
@pytest.mark.parametrize("n", [3, 300, 70000])
def test_preprocess_tile_edges(m, n):
    rng = np.random.default_rng(m * 7 + n)
    _check(rng.integers(0, n, m), rng.integers(0, n, m))


def test_preprocess_shapes():
    i = np.arange(9000)
    _check(np.zeros(9000), np.ones(9000))                             # one edge, drawn 9,000 times
    _check(np.full(9000, 4), np.full(9000, 4))                        # self-loops only
    _check(i, np.full(9000, 9000))                                    # a star
    _check(np.concatenate([np.repeat(np.arange(40), 500), [5000]]),   # 40 hubs without out-edges: a long row gap
           np.concatenate([np.tile(np.arange(100, 600), 40), [5001]]))
    rng = np.random.default_rng(3)
    group = np.repeat(np.arange(50), 100)
    base = rng.integers(0, 50, 20000) * 100
    _check(base + rng.integers(0, 100, 20000), base + rng.integers(0, 100, 20000), group)


@pytest.mark.parametrize("pairs", [3071, 3072, 3073, 4096, 4097])
def test_peel_order_tile_edges(pairs):
    """pairs edges of which some lie in a triangle: e_truss and ptr_truss from
    a sort of one tile, less, and one key more."""
    rng = np.random.default_rng(pairs)
    e = set()
    while len(e) < pairs:
        a, b = rng.integers(0, 400, 2)
        if a != b:
            e.add((min(a, b), max(a, b)))
    rows, cols, rp, verts = O.preprocess(np.array(sorted(e), np.int32), stable=True)
    assert len(cols) == pairs
    V = len(verts)
    kmax, et, pt, truss = O.k_truss(rows, cols, O.tiling_row_ptr(rows, cols, V, 1), V, 1)
    r = T.truss_decompose(CSRCOO(columns=torch.as_tensor(cols).cuda(), row_ptr=torch.as_tensor(rp).long().cuda(),
                                 rows=torch.as_tensor(rows).cuda()))
    assert r.kmax == kmax and np.array_equal(r.e_truss.cpu().numpy(), et)
    assert np.array_equal(r.ptr_truss.cpu().numpy(), pt) and np.array_equal(r.truss.cpu().numpy(), truss)


@pytest.mark.parametrize("m", [(1 << 20) - 1, 1 << 20, (1 << 20) + 1, (1 << 20) + 4095, (1 << 20) + 4097])
def test_preprocess_large_tiles(m):
    """Draws around the size from which the sort takes its larger tiles."""
    rng = np.random.default_rng(m)
    _check(rng.integers(0, 300, m), rng.integers(0, 60000, m))

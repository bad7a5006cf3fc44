"""The drop-in operators over rows at the edges of their walks: more rows than
blocks, rows a block stages whole, rows staged in pieces of 256 keys, -1 holes,
lists of affected edges in any order and of any length; against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import trusstensor as tt

pytestmark = pytest.mark.gpu


def cu(a, dtype=torch.int32):
    return torch.as_tensor(np.ascontiguousarray(a)).to(dtype).cuda()


def _rows_graph(lengths, V, seed):
    """Row i < len(lengths) points at the lengths[i] ids after it, the rest at
    a few random ids above their own."""
    rng = np.random.default_rng(seed)
    r, c = [], []
    for u in range(V):
        if u < len(lengths):
            t = np.arange(u + 1, min(V, u + 1 + lengths[u]))
        else:
            t = np.unique(rng.integers(u + 1, V, 12)) if u + 1 < V else np.empty(0, np.int64)
        r.append(np.full(len(t), u))
        c.append(t)
    rows, cols = np.concatenate(r).astype(np.int32), np.concatenate(c).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=V))]).astype(np.int32)
    return rows, cols, rp


@pytest.mark.parametrize("V", [3, 455, 457, 1025])
def test_support_rows_over_blocks(V):
    lengths = [1, 31, 32, 33, 255, 256, 257, 300, 511, 512, 513, 900]
    rows, cols, rp = _rows_graph(lengths, V, V)
    out = torch.zeros(len(cols), dtype=torch.int32, device="cuda")
    tt.segment_isin2(cu(rows), cu(cols), cu(rp), out)
    assert np.array_equal(out.cpu().numpy(), O.support(rows, cols, rp, 1))


def test_support_many_rows():
    """More rows than one scan of every block, a long one among the last."""
    V, at = 300000, 298000
    hub = np.arange(at + 1, V)
    pairs = np.arange(0, V - 4, 2)
    rows = np.concatenate([pairs, pairs, pairs + 1, np.full(len(hub), at)])
    cols = np.concatenate([pairs + 1, pairs + 2, pairs + 2, hub])
    k = np.unique(rows.astype(np.int64) * V + cols)
    rows, cols = (k // V).astype(np.int32), (k % V).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=V))]).astype(np.int32)
    out = torch.zeros(len(cols), dtype=torch.int32, device="cuda")
    tt.segment_isin2(cu(rows), cu(cols), cu(rp), out)
    assert np.array_equal(out.cpu().numpy(), O.support(rows, cols, rp, 1))


@pytest.fixture(scope="module")
def pieces():
    lengths = [700, 1, 255, 256, 257, 31, 32, 33, 511, 512, 513, 64, 65, 600]
    return _rows_graph(lengths, 800, 5)


@pytest.mark.parametrize("holes", [0.0, 0.3])
@pytest.mark.parametrize("pick", [1, 33, 2500, None])
@pytest.mark.parametrize("kind", ["not", "deleted"])
def test_affected_rows_in_pieces(pieces, kind, pick, holes):
    rows, cols, rp = pieces
    rng = np.random.default_rng(11)
    sup = O.support(rows, cols, rp, 1)
    E = len(cols)
    dead = rng.random(E) < holes
    cols = np.where(dead, -1, cols).astype(np.int32)
    l = max(1, int(np.percentile(sup, 30)))
    mark = ((rng.random(E) < 0.7) & ~dead).astype(np.uint8)
    aff = rng.permutation(np.nonzero(~dead)[0]).astype(np.int32)[:pick]
    if pick is None:
        aff = np.sort(aff)
    o_sup, o_nm = sup.copy(), np.zeros(E, np.uint8)
    g_sup, g_nm = cu(sup), torch.zeros(E, dtype=torch.bool, device="cuda")
    args = (cu(aff), cu(rows), cu(cols), cu(rp), cu(mark, torch.bool), l, g_nm, g_sup)
    if kind == "not":
        O.all_affected_support_tilenot(aff, rows, cols, rp, 1, mark, l, o_nm, o_sup)
        tt.sub_AllAffectedSupport_not(*args)
    else:
        O.all_affected_support_tile(aff, rows, cols, rp, 1, mark, l, o_nm, o_sup)
        tt.sub_AllAffectedSupport(*args)
    g_sup, g_nm = g_sup.cpu().numpy(), g_nm.cpu().numpy().astype(np.uint8)
    assert np.array_equal(g_nm, o_nm)
    hi = (o_sup > l) | (g_sup > l)
    assert np.array_equal(o_sup[hi], g_sup[hi])


def test_edge_walks_in_pieces(pieces):
    rows, cols, rp = pieces
    E = len(cols)
    for k in (3, 100000):
        o = np.zeros(E, np.int32)
        O.segment_isin2tile_k(rows, cols, rp, 1, k, o)
        g = torch.zeros(E, dtype=torch.int32, device="cuda")
        tt.segment_isin2_k(cu(rows), cu(cols), cu(rp), k, g)
        assert np.array_equal(np.minimum(g.cpu().numpy(), k), np.minimum(o, k))
    sup = O.support(rows, cols, rp, 1)
    mark = (np.random.default_rng(2).random(E) < 0.2).astype(np.uint8)
    o = sup.copy()
    O.sub_affected_support_tile(rows, cols, rp, 1, mark, o)
    g = cu(sup)
    tt.sub_AffectedSupport(cu(rows), cu(cols), cu(rp), cu(mark, torch.bool), g)
    assert np.array_equal(g.cpu().numpy(), o)


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_edge_walk_any_alignment(pieces, shift):
    rows, cols, rp = pieces
    buf = torch.full((len(cols) + 8,), 7, dtype=torch.int32, device="cuda")
    c = buf[shift:shift + len(cols)]
    c.copy_(cu(cols))
    g = torch.zeros(len(cols), dtype=torch.int32, device="cuda")
    tt.segment_isin2_k(cu(rows), c, cu(rp), 100000, g)
    assert np.array_equal(g.cpu().numpy(), O.support(rows, cols, rp, 1))

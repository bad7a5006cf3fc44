"""The edge operators on rows far longer than the rows of their heads (a source
of many out-edges that ranks low): the heads' keys are staged and the long row
is streamed.  Around the bounds of that choice, with keys in several pieces,
keys that heads share, -1 holes and any list of edges; against the oracle, and
against plain intersections where it takes two holes for a common column."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tdtdecomposition_gb300 import trusstensor as tt

pytestmark = pytest.mark.gpu
V = 4000


def cu(a, dtype=torch.int32):
    return torch.as_tensor(np.ascontiguousarray(a)).to(dtype).cuda()


def _graph(hub, heads, each, seed):
    """Vertex 0 joined to the `hub` ids after it; the first `heads` of those to
    `each` random ids above their own, a shared one among them."""
    rng = np.random.default_rng(seed)
    r, c = [np.zeros(hub, np.int64)], [np.arange(1, hub + 1)]
    for v in range(1, heads + 1):
        t = np.union1d(rng.choice(np.arange(heads + 1, V - 1), each, replace=False), [V - 1, heads + 1])
        r.append(np.full(len(t), v))
        c.append(t)
    k = np.unique(np.concatenate(r) * V + np.concatenate(c))
    rows, cols = (k // V).astype(np.int32), (k % V).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=V))]).astype(np.int32)
    return rows, cols, rp


def _triangles(rows, cols, rp):
    """(edge, position in N+(v), position in N+(u)) of every common column."""
    out = []
    for u in np.unique(rows):
        at = {int(cols[i]): i for i in range(rp[u], rp[u + 1]) if cols[i] >= 0}
        for e in at.values():
            v = cols[e]
            out += [(e, i, at[int(cols[i])]) for i in range(rp[v], rp[v + 1]) if int(cols[i]) in at]
    return np.array(out, np.int64).reshape(-1, 3)


GRAPHS = {
    "at_row": (512, 40, 3),        # 512 entries are staged in pieces, 513 streamed
    "past_row": (513, 40, 3),
    "at_ratio": (1024, 32, 14),    # 32 heads of 16 keys: half of 1,024, and of 1,025
    "past_ratio": (1026, 32, 14),
    "pieces": (3999, 600, 40),     # 32 heads of some 42 keys: six pieces
    "one_key": (3999, 3000, 0),
}


@pytest.mark.parametrize("holes", [0.0, 0.25])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_long_row_vs_oracle(name, holes):
    rows, cols, rp = _graph(*GRAPHS[name], 3)
    rng = np.random.default_rng(5)
    E = len(cols)
    sup = O.support(rows, cols, rp, 1)
    dead = rng.random(E) < holes
    cols = np.where(dead, -1, cols).astype(np.int32)
    tri = _triangles(rows, cols, rp)
    for k in (2, 100000):
        o = np.bincount(tri.ravel(), minlength=E)
        if holes == 0.0:
            assert np.array_equal(o, sup)
        g = torch.zeros(E, dtype=torch.int32, device="cuda")
        tt.segment_isin2_k(cu(rows), cu(cols), cu(rp), k, g)
        assert np.array_equal(np.minimum(g.cpu().numpy(), k), np.minimum(o, k))
    mark = (rng.random(E) < 0.3).astype(np.uint8)
    m = mark[tri]
    gone = tri[m.any(1)]
    o = sup - np.bincount(gone[mark[gone] == 0], minlength=E)
    g = cu(sup)
    tt.sub_AffectedSupport(cu(rows), cu(cols), cu(rp), cu(mark, torch.bool), g)
    assert np.array_equal(g.cpu().numpy(), o)
    l = 1
    mark = ((rng.random(E) < 0.7) & ~dead).astype(np.uint8)
    for pick in (1, 33, None):
        aff = rng.permutation(np.nonzero(~dead)[0]).astype(np.int32)[:pick]
        if pick is None:
            aff = np.sort(aff)
        for fn, ref in ((tt.sub_AllAffectedSupport_not, O.all_affected_support_tilenot),
                        (tt.sub_AllAffectedSupport, O.all_affected_support_tile)):
            o, o_nm = sup.copy(), np.zeros(E, np.uint8)
            ref(aff, rows, cols, rp, 1, mark, l, o_nm, o)
            g, g_nm = cu(sup), torch.zeros(E, dtype=torch.bool, device="cuda")
            fn(cu(aff), cu(rows), cu(cols), cu(rp), cu(mark, torch.bool), l, g_nm, g)
            g, g_nm = g.cpu().numpy(), g_nm.cpu().numpy().astype(np.uint8)
            assert np.array_equal(g_nm, o_nm)
            hi = (o > l) | (g > l)
            assert np.array_equal(o[hi], g[hi])


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_long_row_any_alignment(shift):
    rows, cols, rp = _graph(3999, 600, 40, 4)
    buf = torch.full((len(cols) + 8,), 7, dtype=torch.int32, device="cuda")
    c = buf[shift:shift + len(cols)]
    c.copy_(cu(cols))
    g = torch.zeros(len(cols), dtype=torch.int32, device="cuda")
    tt.segment_isin2_k(cu(rows), c, cu(rp), 100000, g)
    assert np.array_equal(g.cpu().numpy(), O.support(rows, cols, rp, 1))

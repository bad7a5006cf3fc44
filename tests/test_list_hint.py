"""The triangle count that a workspace remembers sizes the list tail of the next
graph with as many edges and vertices, wherever that lies; it decides nothing
else, and a run that reads its result back corrects it."""
import numpy as np
import pytest
import torch

from tdtdecomposition_gb300 import CSRCOO, batch as B, truss as T

V, K = 600, 100
E = K * (K - 1) // 2


def _csr(rows, cols):
    k = np.sort(rows.astype(np.int64) * V + cols)
    return (torch.as_tensor((k % V).astype(np.int32)),
            torch.as_tensor(np.concatenate([[0], np.cumsum(np.bincount(k // V, minlength=V))])))


def _sparse(seed=1):
    rng = np.random.default_rng(seed)
    a, b = np.triu_indices(V, 1)
    i = rng.choice(len(a), E, replace=False)
    return _csr(a[i], b[i])


def _clique():
    return _csr(*np.triu_indices(K, 1))


def test_hint_is_of_the_size(monkeypatch):
    calls = []
    monkeypatch.setattr(T, "triangle_count_arrays", lambda *a: calls.append(1) or 1000)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (1 << 40, 1 << 40))
    ws = T.Workspace("cpu")
    c, rp = _sparse()
    S = T._stage_room(c, rp)
    assert T.stage_bytes(c, rp) <= S <= T.stage_bytes(c, rp) * 65 // 64
    assert T._list_bytes(ws, c, rp, True, 1 << 20) == 24 * 1000 + 256 + S and calls == [1]
    assert T._list_bytes(ws, c.clone(), rp.clone(), "auto", 1 << 20) == 24 * 1000 + 256 + S and calls == [1]
    # a run found more triangles, then one with more slots than were asked for
    stats = [0] * T.STAT_COUNT
    stats[T.STAT_TRIANGLES] = 5000
    T._learn(ws, c, rp, stats, 24 * 1000 + 256 + S)
    assert T._list_bytes(ws, c, rp, True, 1 << 20) == 24 * 5000 + 256 + S and calls == [1]
    stats[T.STAT_LISTED] = 1
    c2, rp2 = _clique()
    T._learn(ws, c2, rp2, stats, 24 * 5000 + 256 + S)
    S2 = T._stage_room(c2, rp2)
    assert T._list_bytes(ws, c2, rp2, True, 1 << 20) == 24 * 5000 + 256 + S2 and calls == [1]
    # what the workspace has is offered; a capture counts
    ws.buf = torch.empty(1, dtype=torch.uint8).expand(1 << 30)
    assert T._list_bytes(ws, c, rp, "auto", 1 << 20) == (1 << 30) - (1 << 20)
    assert T._list_bytes(ws, c, rp, False, 1 << 20) == 0 and calls == [1]
    T._list_bytes(ws, c, rp, True, 1 << 20, None, count=True)
    assert calls == [1, 1]


def _set(g, c, rp):
    g.columns.copy_(c)
    g.row_ptr.copy_(rp)


@pytest.mark.gpu
def test_refilled_buffers():
    """A graph of few triangles, then a clique in the same buffers."""
    c, rp = _sparse()
    g = CSRCOO(columns=c.cuda(), row_ptr=rp.cuda())
    ws = T.Workspace()
    a = T.truss_decompose(g, workspace=ws, lists=True)
    assert a.listed and a.kmax < K
    _set(g, *_clique())
    r = T.truss_decompose(g, workspace=ws, lists=True)
    assert r.listed and r.kmax == K and r.triangles == K * (K - 1) * (K - 2) // 6 and bool((r.truss == K).all())
    # "auto" may search once, and lists the next time
    ws = T.Workspace()
    _set(g, c, rp)
    first = T.truss_decompose(g, workspace=ws)
    assert torch.equal(first.truss, a.truss) and torch.equal(first.e_truss, a.e_truss)
    _set(g, *_clique())
    for listed in (None, True):
        r = T.truss_decompose(g, workspace=ws)
        assert r.kmax == K and bool((r.truss == K).all()) and listed in (None, r.listed)
    _set(g, c, rp)
    back = T.truss_decompose(g, workspace=ws)
    assert back.listed and torch.equal(back.truss, a.truss)
    assert bool(T.ktruss_search(g, 3, workspace=ws).eq(a.truss >= 3).all())


@pytest.mark.gpu
def test_capture_counts_its_own_graph():
    c, rp = _sparse()
    ws = T.Workspace()
    T.truss_decompose(CSRCOO(columns=c.cuda(), row_ptr=rp.cuda()), workspace=ws)
    c, rp = _clique()
    g = CSRCOO(columns=c.cuda(), row_ptr=rp.cuda())
    cap = B.capture(B.batch_from_union(g, torch.tensor([0, E]), torch.tensor([0, V])), workspace=ws)
    r = cap.replay()
    assert bool((r.truss == K).all()) and int(cap.stats[T.STAT_LISTED]) > 0

"""The list tail that truss_decompose and ktruss_search ask for: lists plus the
staging slots of the one walk, the lists alone where the slots do not fit or
are out of proportion to them (a hub that ranks low), or nothing."""
import numpy as np
import pytest
import torch

from tdtdecomposition_gb300 import CSRCOO, truss as T

GB = 1 << 30


def _wheel(n, dev="cpu"):
    """Hub 0 joined to the n - 1 vertices of a ring."""
    i = np.arange(1, n, dtype=np.int64)
    a, b = np.concatenate([0 * i, i[:-1], [1]]), np.concatenate([i, i[:-1] + 1, [n - 1]])
    k = np.unique(a * n + b)
    rp = np.concatenate([[0], np.cumsum(np.bincount(k // n, minlength=n))])
    return CSRCOO(columns=torch.as_tensor((k % n).astype(np.int32)).to(dev), row_ptr=torch.as_tensor(rp).to(dev))


def _ranked(n, d):
    """n rows of d edges each."""
    cols = (np.arange(n)[:, None] + 1 + np.arange(d)[None]).ravel().astype(np.int32)
    return CSRCOO(columns=torch.as_tensor(cols),
                  row_ptr=torch.as_tensor(np.concatenate([np.arange(n + 1) * d, np.full(d, n * d)])))


@pytest.mark.parametrize("graph,tri,base,free,want", [
    (_ranked(1000, 10), 10000, 1 << 20, 100 * GB, {True: "staged", "auto": "staged", False: "none"}),
    # room for the lists and 0.9 of the slots; for the lists alone; for neither
    (_ranked(1000, 30), 10000, 1 << 20, (1 << 20) + 3000000, {True: "lists", "auto": "lists"}),
    (_ranked(1000, 30), 10000, 1 << 20, (1 << 20) + 4000000, {True: "staged", "auto": "lists"}),
    (_ranked(1000, 30), 10000, 1 << 20, (1 << 20) + 300000, {True: "lists", "auto": "none"}),
    # slots far out of proportion to the lists, whatever the memory
    (_wheel(300000), 299999, 72 << 20, 270 * GB, {True: "lists", "auto": "lists"}),
    (_wheel(300000), 299999, 72 << 20, 900 * GB, {True: "lists", "auto": "lists"}),
])
def test_tail(monkeypatch, graph, tri, base, free, want):
    monkeypatch.setattr(T, "triangle_count_arrays", lambda *a: tri)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (free, free))
    S = T._stage_room(graph.columns, graph.row_ptr)
    tails = {"none": 0, "lists": 24 * tri + 256, "staged": 24 * tri + 256 + S}
    for lists, kind in want.items():
        ws = T.Workspace("cpu")
        assert T._list_bytes(ws, graph.columns, graph.row_ptr, lists, base, graph.rows) == tails[kind], (lists, kind)
        # a workspace that holds all of it is used whatever is free
        ws.buf = torch.empty(1, dtype=torch.uint8).expand(base + tails["staged"])
        if kind != "none" and S < 16 * base:
            assert T._list_bytes(ws, graph.columns, graph.row_ptr, lists, base, graph.rows) == tails["staged"]


@pytest.mark.gpu
@pytest.mark.parametrize("lists", [True, "auto", False])
def test_low_hub_decomposes_with_lists(lists):
    """360 GB of staging slots, more than the device has."""
    n = 300000
    g = _wheel(n, "cuda")
    r = T.truss_decompose(g, workspace=T.Workspace(), lists=lists)
    assert (r.kmax, r.triangles, r.listing) == (3, n - 1, 0 if lists is False else 1)
    assert bool((r.truss == 3).all())
    assert bool(T.ktruss_search(g, 3, workspace=T.Workspace(), lists=lists).all())

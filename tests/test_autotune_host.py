"""The tuner's search with made-up times: it picks the fastest of what a
decomposition depends on, and leaves the wedge width of the support operator,
which it does not depend on, alone."""
import torch

from tdtdecomposition_gb300 import CSRCOO, autotune


class _Knobs:
    def __init__(self):
        self.vec, self.caps, self.grid = None, None, None

    def tdt_set_support_caps(self, w, h):
        self.caps = (w, h)

    def tdt_set_peel_grid(self, n):
        self.grid = n

    def tdt_set_vector_walk(self, on):
        self.vec = on


def _tune(monkeypatch, times, **kw):
    knobs, seen = _Knobs(), []
    monkeypatch.setattr(autotune, "_cache", {})
    monkeypatch.setattr(autotune._lib, "load", lambda: knobs)
    monkeypatch.setattr(autotune.T, "truss_decompose", lambda g, workspace, lists, sync: seen.append(lists))

    def timed(fn, reps=1):
        fn()
        return times(knobs, seen[-1])

    monkeypatch.setattr(autotune, "_time", timed)
    g = CSRCOO(columns=torch.tensor([1, 2], dtype=torch.int32), row_ptr=torch.tensor([0, 2, 2, 2]))
    return autotune.tune(g, **kw), knobs


def test_picks_the_fastest_of_what_matters(monkeypatch):
    cfg, knobs = _tune(monkeypatch, lambda k, lists: 10 - (k.caps == (64, 0)) - 2 * (lists is False) - (k.grid == 2))
    assert tuple(cfg) == (64, 0, False, 2, 1)
    assert (knobs.caps, knobs.grid, knobs.vec) == ((64, 0), 2, 1)


def test_leaves_the_wedge_width(monkeypatch):
    cfg, knobs = _tune(monkeypatch, lambda k, lists: 1.0 if k.vec else 0.5)  # noise in favour of the scalar walk
    assert cfg.vec == 1 and knobs.vec == 1
    cfg, knobs = _tune(monkeypatch, lambda k, lists: 1.0, vec_options=(0,))
    assert cfg.vec == 0 and knobs.vec == 0

"""The edge operators on rows that hold copies of a column: one key of a staged
row is hit more often than 16 bits count."""
import numpy as np
import pytest
import torch

from tdtdecomposition_gb300 import trusstensor as tt

pytestmark = pytest.mark.gpu

U, V1, X, NV = 0, 1, 2, 5


def _graph(copies):
    """u -> {v, x, y, z}, v -> copies of x: the edge (u, v) closes `copies`
    triangles, all of them at (u, x)."""
    rows = np.concatenate([[U] * 4, np.full(copies, V1)])
    cols = np.concatenate([[V1, X, 3, 4], np.full(copies, X)])
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=NV))])
    return tuple(torch.as_tensor(a.astype(np.int32)).cuda() for a in (rows, cols, rp))


@pytest.mark.parametrize("copies", [10, 32767, 32768, 32769, 65535, 65536, 65537, 200003])
def test_copies_are_all_counted(copies):
    rows, cols, rp = _graph(copies)
    want = np.zeros(4 + copies, np.int64)
    want[0] = want[1] = copies
    want[4:] = 1
    out = torch.zeros_like(cols)
    tt.segment_isin2_k(rows, cols, rp, 1 << 30, out)
    assert np.array_equal(out.cpu().numpy(), want)
    # decrements: every edge alive but (u, v), which goes
    out = torch.full_like(cols, copies + 1)
    mark = torch.zeros(4 + copies, dtype=torch.bool, device="cuda")
    mark[0] = True
    tt.sub_AffectedSupport(rows, cols, rp, mark, out)
    got = out.cpu().numpy()
    assert got[1] == 1 and np.array_equal(got[2:4], [copies + 1] * 2) and (got[4:] == copies).all()
    # the peel update stops at its level
    out = torch.full_like(cols, copies + 1)
    n_mark = torch.zeros_like(mark)
    alive = ~mark
    tt.sub_AllAffectedSupport_not(torch.zeros(1, dtype=torch.int32, device="cuda"), rows, cols, rp, alive, 5, n_mark, out)
    got = out.cpu().numpy()
    assert got[1] == max(1, 5) and np.array_equal(got[2:4], [copies + 1] * 2) and (got[4:] == copies).all()
    assert bool(n_mark[1]) and not bool(n_mark[2])

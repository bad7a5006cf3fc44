"""tdt_segment_max against numpy: slab and segment edges, empty segments, and
values outside the segments."""
import numpy as np
import pytest
import torch

from tdtdecomposition_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nseg,hi", [(1, 1), (1, 200001), (3, 129), (512, 700), (5000, 3), (40, 100003)])
def test_segment_max(nseg, hi):
    rng = np.random.default_rng(nseg + hi)
    off = np.concatenate([[0], np.cumsum(rng.integers(0, hi + 1, nseg))]).astype(np.int64)
    n = int(off[-1]) + 5  # values past the last segment are ignored
    vals = rng.integers(-(1 << 31), 1 << 31, n).astype(np.int32)
    want = np.full(nseg, -7, np.int64)
    for g in range(nseg):
        if off[g + 1] > off[g]:
            want[g] = max(want[g], int(vals[off[g]:off[g + 1]].max()))
    out = torch.full((nseg,), -7, dtype=torch.int64, device="cuda")
    v, o = torch.from_numpy(vals).cuda(), torch.from_numpy(off).cuda()
    rc = _lib.load().tdt_segment_max(v.data_ptr(), n, o.data_ptr(), nseg, out.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert np.array_equal(out.cpu().numpy(), want)

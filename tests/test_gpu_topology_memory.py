"""From 2^24 cells on, a topology holds arrays for the exits that the raster has (a row that drains east has one per
tile boundary), not for the most that its shape could have.  Accu of ones along the rows is exact below 2^24."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, cols", [(4096, 4096), (4099, 4161)])
def test_exit_arrays(rows, cols):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework as lfr
    a = lfr.from_numpy(np.full((rows, cols), 6, np.uint8))
    s = a.topology().stats()
    trows, tcols = -(-rows // 64), -(-cols // 64)
    assert s["tile_exits"] == rows * (tcols - 1)
    # per cell 7 bytes and 5 of scratch; per tile two tables of 2 bytes a cell, 1 KB of inflows and a few words; per exit
    # 24 bytes, 24 of scratch and its share of the scan's blocks
    most = 12 * rows * cols + trows * tcols * (4 * 4096 + 1024 + 64) + 50 * s["tile_exits"] + 2 ** 16
    assert s["device_bytes"] <= most
    got = lfr.accu(a, lfr.from_numpy(np.ones((rows, cols), np.float32))).data
    want = torch.arange(1, cols + 1, device=got.device, dtype=torch.float32).expand(rows, cols)
    assert torch.equal(got, want)

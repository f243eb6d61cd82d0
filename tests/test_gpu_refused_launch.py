"""accu (float32) on small rasters after a call of which a launch was refused: the call fails, and the next ones on that
handle give the same bits as before it.  (Sizes with the exits' scan in the first pass and in a launch of its own.)"""
import numpy as np
import pytest

from lue_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(255, 301), (1000, 1024)])
def test_calls_after_a_refused_launch(monkeypatch, shape):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework as lfr
    a = lfr.from_numpy(synthetic.flow_direction(*shape, 7, 60.0, wavelength=max(shape) / 2))
    m = np.random.default_rng(7).lognormal(0.0, 1.0, shape).astype(np.float32)
    x, other = lfr.from_numpy(m), lfr.from_numpy((1.75 * m).astype(np.float32))
    want = [lfr.to_numpy(lfr.accu(a, y)) for y in (x, other)]
    monkeypatch.setenv("LUE_GB300_TILE_REFUSE", "1")
    with pytest.raises(RuntimeError):
        lfr.accu(a, other)
    monkeypatch.delenv("LUE_GB300_TILE_REFUSE")
    for _ in range(2):
        for y, w in zip((x, other), want):
            assert np.array_equal(lfr.to_numpy(lfr.accu(a, y)), w, equal_nan=True)

"""The path engine on a raster whose first level above 0 is large (about 7 % of the cells, 2^18 and more: two positions per
thread, one chunk per CTA), with paths that cross chunks and with look-back on every level.

Tolerance: the inputs are whole numbers, whose sums and differences are exact in float-float, so float32 results
equal the float64 oracle's rounded to float32; float64 sums are exact."""
import numpy as np
import pytest

from lue_gb300 import synthetic
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


@pytest.fixture(scope="module")
def raster():
    shape = (2600, 2701)
    fd = synthetic.flow_direction(*shape, 17, 60.0, wavelength=1300).copy()
    rng = np.random.default_rng(17)
    fd[rng.random(shape) < 0.0005] = 255
    m = rng.integers(0, 4, shape).astype(np.float32)
    b = rng.integers(0, 12, shape).astype(np.float32)
    m[rng.random(shape) < 0.0005] = np.nan
    return fd, m, b


@pytest.mark.parametrize("longest", [None, "0"], ids=["default", "look-back on every level"])
@pytest.mark.parametrize("op", ["threshold", "capacity", "trigger", "accu"])
def test_large_levels(lfr, raster, monkeypatch, op, longest):
    if longest:
        monkeypatch.setenv("LUE_GB300_PATH_FREE_LONGEST", longest)
    fd, m, b = raster
    a = lfr.from_numpy(fd)
    m64, b64 = m.astype(np.float64), b.astype(np.float64)
    if op == "accu":
        got, want = [lfr.accu(a, lfr.from_numpy(m64))], [oracle.accu(fd, m64, fd.shape, dtype=np.float64)]
    else:
        got = getattr(lfr, f"accu_{op}")(a, lfr.from_numpy(m), lfr.from_numpy(b))
        want = [x.astype(np.float32) for x in getattr(oracle, f"accu_{op}")(fd, m64, b64, fd.shape, dtype=np.float64)]
    for g, w in zip(got, want):
        assert np.array_equal(lfr.to_numpy(g), w, equal_nan=True)

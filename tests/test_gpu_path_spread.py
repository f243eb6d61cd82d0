"""Path engine calls whose results are spread over the raster: accu_fraction on large levels, a look-back whose waits give
up, and the raster size from which it is the default.

Tolerances: whole numbers and redone calls bit for bit; accu_fraction that of the float32 operations against the float64
oracle."""
import numpy as np
import pytest

from lue_gb300 import synthetic
from oracle import oracle
from tests import parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


@pytest.fixture(scope="module")
def raster():
    shape = (2893, 2907)  # beyond 2^23 cells
    fd = synthetic.flow_direction(*shape, 19, 60.0, wavelength=1300).copy()
    rng = np.random.default_rng(19)
    fd[rng.random(shape) < 0.0005] = 255
    m = rng.integers(0, 4, shape).astype(np.float32)
    m[rng.random(shape) < 0.0005] = np.nan
    return fd, m, rng.integers(0, 12, shape).astype(np.float32), rng.random(shape, dtype=np.float32)


def _call(lfr, raster, op):
    fd, m, b, f = raster
    a = lfr.from_numpy(fd)
    got = getattr(lfr, f"accu_{op}")(a, lfr.from_numpy(m), lfr.from_numpy(f if op == "fraction" else b))
    return a, [lfr.to_numpy(x) for x in got]


@pytest.mark.parametrize("hook", [None, ("SPREAD", str(1 << 40)), ("FREE_LONGEST", "0")], ids=["default", "straight", "look-back"])
def test_fraction(lfr, raster, monkeypatch, hook):
    if hook:
        monkeypatch.setenv("LUE_GB300_PATH_" + hook[0], hook[1])
    fd, m, _, f = raster
    want = oracle.accu_fraction(fd, m.astype(np.float64), f.astype(np.float64), fd.shape, dtype=np.float64)
    for g, w, name in zip(_call(lfr, raster, "fraction")[1], want, ("outflow", "remainder")):
        parity.assert_close32(g, w, name)


@pytest.mark.parametrize("op", ["threshold", "capacity"])
def test_default_size_and_waits_that_give_up(lfr, raster, monkeypatch, op):
    fd, m, b, _ = raster
    want = getattr(oracle, f"accu_{op}")(fd, m.astype(np.float64), b.astype(np.float64), fd.shape, dtype=np.float64)
    want = [w.astype(np.float32) for w in want]
    a, got = _call(lfr, raster, op)
    assert a.topology().stats()["device_bytes"] >= 32 * fd.size  # the results by position are there
    for g, w in zip(got, want):
        assert np.array_equal(g, w, equal_nan=True)
    monkeypatch.setenv("LUE_GB300_PATH_FREE_LONGEST", "0")
    monkeypatch.setenv("LUE_GB300_PATH_POLLS", "0")
    for g, w in zip(_call(lfr, raster, op)[1], want):
        assert np.array_equal(g, w, equal_nan=True)

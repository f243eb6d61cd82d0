"""Float32 accu_trigger on the path engine: the composed maps against the walk engine and the float64 oracle.

A cell's outflow jumps at its trigger, so inputs are chosen where both engines' totals are on the same side:
whole numbers, whose float-float sums are exact (results equal bit for bit, ties with the trigger included),
and continuous values, where a total within rounding of its trigger does not occur (float-float carries about
48 bits, the values 24): those agree within the float32 tolerance of the other rules."""
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


def _raster(shape, seed, amplitude=40.0, wavelength=None):
    fd = synthetic.flow_direction(*shape, seed, amplitude, wavelength=wavelength or max(shape) / 2).copy()
    rng = np.random.default_rng(seed)
    fd[rng.random(shape) < 0.001] = 255
    return fd, rng


def _run(lfr, fd, m, b):
    arg = lambda x: x if np.isscalar(x) else lfr.from_numpy(x)  # noqa: E731
    return [lfr.to_numpy(x) for x in lfr.accu_trigger(lfr.from_numpy(fd), arg(m), arg(b))]


SHAPES = [(1, 1), (1, 300), (300, 1), (65, 31), (333, 777), (1024, 1024)]


@pytest.mark.parametrize("longest", [None, "0"], ids=["default", "look-back on every level"])
@pytest.mark.parametrize("shape", SHAPES)
def test_whole_numbers_equal_the_walk_engine(lfr, monkeypatch, shape, longest):
    if longest:
        monkeypatch.setenv("LUE_GB300_PATH_FREE_LONGEST", longest)
    fd, rng = _raster(shape, 91)
    m = rng.integers(0, 4, shape).astype(np.float32)
    b = rng.integers(0, 12, shape).astype(np.float32)
    m[rng.random(shape) < 0.001] = np.nan
    m[rng.random(shape) < 0.001] = -1.0
    b[rng.random(shape) < 0.0005] = np.nan
    got = _run(lfr, fd, m, b)
    monkeypatch.setenv("LUE_GB300_ENGINE", "walk")
    for g, w in zip(got, _run(lfr, fd, m, b)):
        assert np.array_equal(g, w, equal_nan=True)


@pytest.mark.parametrize("scale", [0.5, 3.0, 400.0])
def test_long_paths_against_the_oracle(lfr, scale):
    fd, rng = _raster((2048, 1531), 93, amplitude=200.0, wavelength=2048)
    m = rng.lognormal(0.0, 1.0, fd.shape).astype(np.float32)
    b = (scale * rng.lognormal(0.0, 1.0, fd.shape)).astype(np.float32)
    want = oracle.accu_trigger(fd, m.astype(np.float64), b.astype(np.float64), fd.shape, dtype=np.float64)
    for g, w, name in zip(_run(lfr, fd, m, b), want, ("outflow", "remainder")):
        parity.assert_close32(g, w, name)


def test_scalars_and_infinities(lfr, monkeypatch):
    fd, rng = _raster((150, 170), 95)
    m = rng.integers(0, 4, fd.shape).astype(np.float32)
    inf = m.copy()
    inf[40, 50] = np.inf
    b = np.full(fd.shape, 7.0, np.float32)
    b[60:70] = np.inf  # never reached
    cases = [(m, 5.0), (2.0, b), (1.0, 3.0), (inf, b)]
    got = [_run(lfr, fd, *c) for c in cases]
    monkeypatch.setenv("LUE_GB300_ENGINE", "walk")
    for g, c in zip(got, cases):
        for x, y in zip(g, _run(lfr, fd, *c)):
            assert np.array_equal(x, y, equal_nan=True)

"""The path engine on a raster whose first level above 0 is large (about 7 % of the cells, 2^18 and more: two positions per
thread, one chunk per CTA), with paths that cross chunks, with look-back on every level and with the results
collected by position and spread over the raster (the default from 2^23 cells on).

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


def _check(lfr, fd, m, b, op):
    a = lfr.from_numpy(fd)
    m64, b64 = m.astype(np.float64), b.astype(np.float64)
    if op == "accu":
        got, want = [lfr.accu(a, lfr.from_numpy(m64))], [oracle.accu(fd, m64, fd.shape, dtype=np.float64)]
    else:
        got = getattr(lfr, f"accu_{op}")(a, lfr.from_numpy(m), lfr.from_numpy(b))
        want = [x.astype(np.float32) for x in getattr(oracle, f"accu_{op}")(fd, m64, b64, fd.shape, dtype=np.float64)]
    for g, w in zip(got, want):
        assert np.array_equal(lfr.to_numpy(g), w, equal_nan=True)


@pytest.mark.parametrize("hook", [None, ("FREE_LONGEST", "0"), ("SPREAD", "0")],
                         ids=["default", "look-back on every level", "results spread"])
@pytest.mark.parametrize("op", ["threshold", "capacity", "trigger", "accu"])
def test_large_levels(lfr, raster, monkeypatch, op, hook):
    if hook:
        monkeypatch.setenv("LUE_GB300_PATH_" + hook[0], hook[1])
    _check(lfr, *raster, op)


@pytest.mark.parametrize("shape", [(1, 1), (1, 300), (300, 1), (64, 64), (65, 63), (129, 320)])
def test_results_spread_over_tile_edges(lfr, monkeypatch, shape):
    monkeypatch.setenv("LUE_GB300_PATH_SPREAD", "0")
    fd = synthetic.flow_direction(*shape, 5, 20.0, wavelength=max(shape) / 2).copy()
    rng = np.random.default_rng(5)
    fd[rng.random(shape) < 0.02] = 255
    _check(lfr, fd, rng.integers(0, 4, shape).astype(np.float32), rng.integers(0, 12, shape).astype(np.float32), "threshold")


def test_spread_results_captured_in_a_graph(lfr, monkeypatch):
    import torch
    monkeypatch.setenv("LUE_GB300_PATH_SPREAD", "0")
    fd = synthetic.flow_direction(333, 777, 5, 20.0, wavelength=400)
    rng = np.random.default_rng(5)
    a = lfr.from_numpy(fd)
    m, b = (lfr.from_numpy(rng.integers(0, k, fd.shape).astype(np.float32)) for k in (4, 12))
    want = [lfr.to_numpy(x) for x in lfr.accu_threshold(a, m, b)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = lfr.accu_threshold(a, m, b)
    for _ in range(2):
        g.replay()
        for x, w in zip(got, want):
            assert np.array_equal(lfr.to_numpy(x), w, equal_nan=True)

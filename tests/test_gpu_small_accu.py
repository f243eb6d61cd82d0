"""accu (float32) where its launches change with the raster's size: one tile, tiles without exits, up to 4096 exits (their
scan is done by the last CTA of the first pass), more exits, the last size with overlapping launches (1024 tiles)
and the first without; calls that the walk engine redoes, between normal ones; a captured graph.

Tolerance: that of every float32 accu test (1e-5 relative against the float64 oracle); repeated, captured and
redone calls are compared bit for bit."""
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


def _raster(shape, seed):
    fd = synthetic.flow_direction(*shape, seed, 60.0, wavelength=max(shape) / 2).copy()
    rng = np.random.default_rng(seed)
    fd[rng.random(shape) < 0.001] = 255
    m = rng.lognormal(0.0, 1.0, shape).astype(np.float32)
    m[rng.random(shape) < 0.0005] = np.nan
    return fd, m


@pytest.mark.parametrize("shape", [(1, 1), (64, 64), (65, 64), (64, 700), (255, 301), (384, 512), (1000, 1024),
                                   (2048, 2048), (2048, 2049)])
def test_sizes(lfr, monkeypatch, shape):
    fd, m = _raster(shape, 7)
    a = lfr.from_numpy(fd)
    normal = lfr.from_numpy(m)
    inf = m.copy()
    inf[shape[0] // 2, shape[1] // 2] = np.inf
    big = lfr.from_numpy(inf)
    got = [lfr.to_numpy(lfr.accu(a, x)) for x in (normal, big, normal, normal, big)]
    parity.assert_close32(got[0], oracle.accu(fd, m.astype(np.float64), fd.shape, dtype=np.float64), f"accu {shape}")
    assert np.array_equal(got[0], got[2], equal_nan=True) and np.array_equal(got[0], got[3], equal_nan=True)
    monkeypatch.setenv("LUE_GB300_ENGINE", "walk")
    walk = lfr.to_numpy(lfr.accu(a, big))
    assert np.array_equal(got[1], walk, equal_nan=True) and np.array_equal(got[4], walk, equal_nan=True)


@pytest.mark.parametrize("shape", [(255, 301), (1000, 1024)])
def test_captured_in_a_graph(lfr, shape):
    import torch
    fd, m = _raster(shape, 9)
    a, x = lfr.from_numpy(fd), lfr.from_numpy(m)
    want = lfr.to_numpy(lfr.accu(a, x))
    other = lfr.from_numpy((2.0 * m).astype(np.float32))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        first, second = lfr.accu(a, x), lfr.accu(a, other)
    for _ in range(3):
        g.replay()
    assert np.array_equal(lfr.to_numpy(first), want, equal_nan=True)
    assert np.array_equal(lfr.to_numpy(second), lfr.to_numpy(lfr.accu(a, other)), equal_nan=True)

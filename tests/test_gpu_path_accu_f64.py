"""Float64 accu on the path engine.  Every sum is of terms >= 0 (no cancellation), and the sum of a path is taken
in blocks, so its relative error against the float64 oracle stays below (number of additions along a path) x
2^-53; the paths here have fewer than 4096 cells: 4096 x 2^-53 = 4.6e-13."""
import numpy as np
import pytest

from lue_gb300 import synthetic
from oracle import oracle

pytestmark = pytest.mark.gpu

RTOL = 4096 * 2.0 ** -53


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


def _check(got, want):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= RTOL * np.abs(want[ok]))


@pytest.mark.parametrize("longest", [None, "0"], ids=["default", "look-back on every level"])
@pytest.mark.parametrize("shape", [(1, 1), (1, 300), (300, 1), (65, 31), (333, 777), (2048, 1531)])
def test_accu_f64_against_the_oracle(lfr, monkeypatch, shape, longest):
    if longest:
        monkeypatch.setenv("LUE_GB300_PATH_FREE_LONGEST", longest)
    fd = synthetic.flow_direction(*shape, 97, 200.0, wavelength=max(shape)).copy()
    rng = np.random.default_rng(97)
    fd[rng.random(shape) < 0.001] = 255
    # thirty decades of material: a sum of tiny terms next to a large river keeps its own precision
    m = rng.lognormal(0.0, 1.0, shape) * 10.0 ** rng.integers(-30, 1, shape)
    m[rng.random(shape) < 0.001] = np.nan
    m[rng.random(shape) < 0.001] = -1.0
    m[rng.random(shape) < 0.01] = 0.0
    got = lfr.to_numpy(lfr.accu(lfr.from_numpy(fd), lfr.from_numpy(m)))
    _check(got, oracle.accu(fd, m, shape, dtype=np.float64))


def test_scalar_and_infinite_material(lfr, monkeypatch):
    shape = (150, 170)
    fd = synthetic.flow_direction(*shape, 99, 40.0)
    m = np.random.default_rng(99).random(shape)
    m[40, 50] = np.inf
    a = lfr.from_numpy(fd)
    got = [lfr.to_numpy(lfr.accu(a, x)) for x in (np.float64(0.25), lfr.from_numpy(m))]
    _check(got[0], oracle.accu(fd, 0.25, shape, dtype=np.float64))
    monkeypatch.setenv("LUE_GB300_ENGINE", "walk")
    assert np.array_equal(got[1], lfr.to_numpy(lfr.accu(a, lfr.from_numpy(m))), equal_nan=True)

"""The nested float-float solve for beta = 3/5 against the float64 oracle over the ranges in which the oracle's
ten Newton steps converge: small and large discharges, rivers far above and far below the local discharge, alpha
from small to large, no-data and negative inflow, one step and several, CTAs of one and of two warps.

Tolerance: the solve keeps about 2^-46 per cell (1.5e-14), and what a cell is off flows on; with at most 97 cells
on a path the sum stays below 97 x 1.5e-14 = 1.5e-12."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

RTOL = 1.5e-12


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


@pytest.mark.parametrize("threads", ["32", "64"])
@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("low, high", [(1e-9, 1e-3), (1e2, 1e9)])
def test_ranges_against_the_oracle(lfr, monkeypatch, low, high, steps, threads):
    monkeypatch.setenv("LUE_GB300_STAGE_THREADS", threads)
    rng = np.random.default_rng(int(steps * 1000 + 7))
    rows, cols = 61, 97
    fd = np.full((rows, cols), 6, np.uint8)  # rows that drain east, joined by diagonals here and there
    fd[1:, :][rng.random((rows - 1, cols)) < 0.1] = 9
    q = np.exp(rng.uniform(np.log(low), np.log(high), fd.shape))
    lat = (rng.random(fd.shape) * 5e-5).astype(np.float32)
    lat[rng.random(fd.shape) < 0.3] = 0.0
    alpha = np.exp(rng.uniform(np.log(1e-3), np.log(1e3), fd.shape)).astype(np.float32)
    q[5, 40] = np.nan
    lat[9, 9] = -1e-6
    alpha[20, 3] = np.nan
    a = lfr.from_numpy(fd)
    args = (lfr.from_numpy(q), lfr.from_numpy(lat), lfr.from_numpy(alpha), 0.6, 3600.0, 100.0)
    got = lfr.to_numpy(lfr.kinematic_wave(a, *args) if steps == 1 else lfr.kinematic_wave_steps(a, *args, steps))
    lat[9, 9] = np.nan  # the multi-step form's domain: negative lateral inflow is no-data in both
    want = q
    for _ in range(steps):
        want = oracle.kinematic_wave(fd, want, lat.astype(np.float64), alpha.astype(np.float64), 0.6, 3600.0, 100.0,
                                     fd.shape, dtype=np.float64)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= RTOL * np.maximum(np.abs(want[ok]), 1e-30))

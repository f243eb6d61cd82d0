"""One step of the beta = 3/5 solve cell by cell against extended precision: cells alone, and cells with one upstream cell.

Tolerances: the last Newton step divides by a float derivative with at most six roundings (6 x 2^-24 = 3.6e-7), from a root
within 1.2e-7; five times their product goes into the discharge: 2.2e-13.  The errors are of both signs: their
mean stays below 2^-48 = 3.6e-15, the size of the products of low parts that the float-float terms leave out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELL, MEAN = 2.2e-13, 2.0 ** -48


def _solve(k, alpha, known):
    y = np.minimum((known / k) ** (np.longdouble(1) / 5), (known / alpha) ** (np.longdouble(1) / 3))
    for _ in range(12):
        y2 = y * y
        y = y - (y * y2 * (k * y2 + alpha) - known) / (y2 * (5 * k * y2 + 3 * alpha))
    return y ** 5


@pytest.mark.parametrize("low, high", [(1e-9, 1e-3), (1e-2, 1e3), (1e2, 1e9)])
@pytest.mark.parametrize("dt, dx", [(3600.0, 100.0), (900.0, 37.0)])
@pytest.mark.parametrize("upstream", [False, True])
def test_cells(upstream, dt, dx, low, high):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework as lfr
    rng = np.random.default_rng(5)
    shape = (256, 512)
    fd = np.full(shape, 5, np.uint8)
    if upstream:
        fd[:, 0::2] = 6
    q = np.exp(rng.uniform(np.log(low), np.log(high), shape))
    lat = (rng.random(shape) * 5e-5).astype(np.float32)
    alpha = np.exp(rng.uniform(np.log(1e-3), np.log(1e3), shape)).astype(np.float32)
    got = lfr.to_numpy(lfr.kinematic_wave(*map(lfr.from_numpy, (fd, q, lat, alpha)), 0.6, dt, dx)).astype(np.longdouble)
    k, a = np.longdouble(dt) / np.longdouble(dx), alpha.astype(np.longdouble)
    known = a * q.astype(np.longdouble) ** (np.longdouble(3) / 5) + np.longdouble(dt) * lat.astype(np.longdouble)
    if upstream:
        known[:, 1::2] += k * _solve(k, a[:, 0::2], known[:, 0::2])
    error = ((got - (want := _solve(k, a, known))) / want).astype(np.float64)
    assert np.abs(error).max() <= (2 if upstream else 1) * CELL  # the upstream cell's error flows on
    assert abs(error.mean()) <= MEAN

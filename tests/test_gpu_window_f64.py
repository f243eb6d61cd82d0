"""float64 upstream and d8_flow_direction, which find their upstream values and compare their drops by integer operations: signs
of zero, infinities of both signs, NaN, cells with eight inflows, equal and tiny drops; bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

VALUES = [0.0, -0.0, 1.5, -1.5, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1e308, -1e308, 1.0 + 2.0 ** -52, 1.0]


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


def _values(shape, p_plain):
    rng = np.random.default_rng(shape[1])
    x = rng.choice(np.array(VALUES), shape)
    plain = rng.random(shape) < p_plain
    x[plain] = rng.normal(0.0, 3.0, shape)[plain]
    return x, rng


def _same(got, want):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok].view(np.int64), want[ok].view(np.int64))


@pytest.mark.parametrize("p_plain", [0.3, 0.95])
@pytest.mark.parametrize("shape", [(3, 3), (9, 31), (33, 250), (64, 515)])
def test_upstream(lfr, shape, p_plain):
    m, rng = _values(shape, p_plain)
    fd = rng.integers(1, 10, shape).astype(np.uint8)
    # a cell in nine has the eight around it draining into it
    around = np.array([[3, 2, 1], [6, 5, 4], [9, 8, 7]], np.uint8)
    r, c = shape[0] // 3 * 3, shape[1] // 3 * 3
    fd[:r, :c] = np.where(rng.random((r, c)) < 0.9, np.tile(around, (r // 3, c // 3)), fd[:r, :c])
    got = lfr.to_numpy(lfr.upstream(lfr.from_numpy(fd), lfr.from_numpy(m)))
    _same(got, oracle.upstream(fd, m, np.float64))


@pytest.mark.parametrize("p_plain", [0.3, 0.95])
@pytest.mark.parametrize("shape", [(1, 1), (3, 3), (9, 31), (33, 250), (64, 515)])
def test_d8(lfr, shape, p_plain):
    z, _ = _values(shape, p_plain)
    assert np.array_equal(lfr.to_numpy(lfr.d8_flow_direction(lfr.from_numpy(z))), oracle.d8_flow_direction(z))

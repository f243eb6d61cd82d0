"""upstream, downstream and d8_flow_direction on shapes around the edges of their windows (30 columns per
warp, 240 per CTA, 8 rows), bit for bit against the oracle: sums are taken in the oracle's neighbour order,
so no tolerance is needed."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 31), (7, 30), (8, 29), (9, 61), (17, 239), (16, 240), (23, 241), (64, 515)]


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_one_hop_operations(lfr, shape, dtype):
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    fd = rng.integers(0, 12, shape).astype(np.uint8)  # directions, sinks and codes that are none
    fd[rng.random(shape) < 0.05] = 255
    m = rng.normal(0.0, 3.0, shape).astype(dtype)
    m[rng.random(shape) < 0.02] = np.nan
    m[rng.random(shape) < 0.01] = np.inf
    a, x = lfr.from_numpy(fd), lfr.from_numpy(m)
    for gpu, cpu in ((lfr.upstream, oracle.upstream), (lfr.downstream, oracle.downstream)):
        assert np.array_equal(lfr.to_numpy(gpu(a, x)), cpu(fd, m, dtype), equal_nan=True)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_d8_flow_direction(lfr, shape, dtype):
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    z = rng.integers(-3, 9, shape).astype(dtype)  # equal drops, and ground below the halo's
    z[rng.random(shape) < 0.05] = np.nan
    assert np.array_equal(lfr.to_numpy(lfr.d8_flow_direction(lfr.from_numpy(z))), oracle.d8_flow_direction(z))

"""Rasters with flow cycles: their levels and statistics come from the tile build too.  Cycles of two cells, inside a tile,
over tile corners and edges, through many tiles, several in one tile, with long tails, at ragged edges and in dense
random codes; accu over them; and no memory held for tile structures that they do not have.

Tolerance: levels and counts are whole numbers and equal the oracle's; accu of ones is exact below 2^24."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


def _ring(fd, r0, c0, r1, c1):
    """A clockwise ring along the rectangle's edge; what lies inside flows north into it."""
    fd[r0:r1 + 1, c0:c1 + 1] = 8
    fd[r0, c0:c1] = 6
    fd[r0:r1, c1] = 2
    fd[r1, c0 + 1:c1 + 1] = 4
    fd[r0 + 1:r1 + 1, c0] = 8
    return fd


def _east(rows, cols):
    return np.full((rows, cols), 6, np.uint8)


def _tails():
    fd = _east(70, 500)  # every row ends in a pair of cells that drain into each other
    fd[:, -1] = 4
    return fd


RASTERS = {
    "pair": np.array([[6, 4]], np.uint8),
    "pair_over_tiles": np.concatenate([_east(1, 64), np.full((1, 64), 4, np.uint8)], axis=1),
    "in_tile": _ring(_east(64, 64), 10, 10, 13, 20),
    "whole_tile": _ring(_east(64, 64), 0, 0, 63, 63),
    "tile_corner": _ring(_east(130, 140), 63, 63, 64, 64),
    "tile_edge": _ring(_east(130, 140), 60, 10, 70, 50),
    "many_tiles": _ring(_east(300, 421), 5, 7, 290, 400),
    "nested": _ring(_ring(_east(200, 200), 10, 10, 180, 190), 70, 70, 90, 100),
    "two_in_a_tile": _ring(_ring(_east(64, 64), 2, 2, 5, 5), 20, 30, 40, 60),
    "ragged": _ring(_east(65, 67), 60, 60, 64, 66),
    "tails": _tails(),
    **{f"random_{k}": np.random.default_rng(k).choice(np.array([1, 2, 3, 4, 6, 7, 8, 9, 5, 255], np.uint8), (190 + k, 257),
                                                      p=[.13] * 4 + [.1] * 4 + [.04] * 2) for k in range(3)},
}


@pytest.mark.parametrize("name", RASTERS)
def test_levels_and_accu(lfr, name):
    fd = RASTERS[name]
    a = lfr.from_numpy(fd)
    level = oracle.downstream_level(fd)
    assert np.array_equal(lfr.to_numpy(lfr.downstream_level(a)), level)
    s = a.topology().stats()
    valid = fd != 255
    assert (level[valid] < 0).any()
    assert s["cycle_cells"] == (valid & (level < 0)).sum()
    assert s["valid_cells"] == valid.sum()
    assert s["ridge_cells"] == (valid & (lfr.to_numpy(lfr.inflow_count(a)) == 0)).sum()
    assert s["max_level"] == max(int(level.max()), 0)
    assert s["tile_exits"] == 0
    # flow directions, counts, masks and levels; counters and residuals; a few bytes for alignment
    assert s["device_bytes"] <= 12 * fd.size + 8 * 256
    got = lfr.to_numpy(lfr.accu(a, lfr.from_numpy(np.ones(fd.shape, np.float32))))
    want = oracle.accu(fd, 1.0, fd.shape, dtype=np.float64)
    reached = valid & (level >= 0)
    assert np.array_equal(got[reached], want[reached].astype(np.float32))

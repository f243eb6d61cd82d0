"""The topology build: inflow counts, downstream levels, statistics and the exit forest (through accu), where the build
over tiles can go wrong (one cell, exact and ragged tiles, one row or column, a path through every cell of a tile and
through every tile, no exits at all, dense random codes) and where it hands over to the walk (cycles inside a
tile, across tiles).

Tolerance: counts, levels and statistics are whole numbers and equal; accu of ones is exact below 2^24.  The counts and
sums are numpy's (the reference's count of a no-data cell depends on the order in which its neighbours are visited
where a flow enters it from below)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

OFFSETS = {7: (-1, -1), 8: (-1, 0), 9: (-1, 1), 4: (0, -1), 6: (0, 1), 1: (1, -1), 2: (1, 0), 3: (1, 1)}


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


def _snake(rows, cols):
    fd = np.full((rows, cols), 6, np.uint8)
    fd[1::2] = 4
    fd[0::2, -1] = 2
    fd[1::2, 0] = 2
    return fd


def _random(rows, cols, codes, seed=3):
    return np.random.default_rng(seed).choice(np.array(codes, np.uint8), (rows, cols))


def _cycle(fd, r, c):
    fd = fd.copy()
    fd[r, c], fd[r, c + 1], fd[r + 1, c + 1], fd[r + 1, c] = 6, 2, 4, 8
    return fd


RASTERS = {
    "cell": np.array([[5]], np.uint8),
    "cell_out": np.array([[6]], np.uint8),
    "no_data": np.full((70, 70), 255, np.uint8),
    "sinks": np.full((65, 63), 5, np.uint8),
    "row": np.full((1, 1000), 6, np.uint8),
    "column": np.full((1000, 1), 8, np.uint8),
    "tile": _random(64, 64, [6, 3, 2, 5, 255]),
    "ragged": _random(65, 63, [6, 3, 2, 1, 5, 255, 77]),
    "dense": _random(200, 333, [6, 3, 2]),
    "up": _random(257, 129, [4, 7, 8, 9, 0]),
    "snake_tile": _snake(64, 64),
    "snake": _snake(131, 300),
    "many_tiles": _random(2112, 1000, [6, 3, 2, 9, 255], 5),
    "cycle_in_tile": _cycle(_random(130, 130, [6, 3, 2, 255]), 20, 20),
    "cycle_over_tiles": _cycle(_random(130, 130, [6, 3, 2, 255]), 63, 63),
    "cycles": _random(150, 150, [1, 2, 3, 4, 5, 6, 7, 8, 9, 255]),
}


def _count_and_accu(fd, level):
    """Inflow counts, outlets, and the accu of ones by level (cells on or below a cycle are not reached)."""
    rows, cols = fd.shape
    down = np.full(fd.shape, -1, np.int64)
    outlets = 0
    for code, (dr, dc) in OFFSETS.items():
        r, c = np.nonzero(fd == code)
        ok = (r + dr >= 0) & (r + dr < rows) & (c + dc >= 0) & (c + dc < cols)
        outlets += int((~ok).sum())
        down[r[ok], c[ok]] = (r[ok] + dr) * cols + c[ok] + dc
    down, level, valid = down.ravel(), level.ravel(), fd.ravel() != 255
    count = np.bincount(down[down >= 0], minlength=fd.size)
    accu = np.where(valid, 1.0, np.nan)
    order = np.flatnonzero(level >= 0)
    order = order[np.argsort(level[order], kind="stable")]
    for cells in np.split(order, np.flatnonzero(np.diff(level[order])) + 1):
        cells = cells[down[cells] >= 0]
        np.add.at(accu, down[cells], accu[cells])
    return np.where(valid, count, 255).reshape(fd.shape), outlets, accu.reshape(fd.shape)


@pytest.mark.parametrize("name", RASTERS)
def test_build(lfr, name):
    fd = RASTERS[name]
    a = lfr.from_numpy(fd)
    level = oracle.downstream_level(fd)
    count, outlets, accu = _count_and_accu(fd, level)
    assert np.array_equal(lfr.to_numpy(lfr.inflow_count(a)), count)
    assert np.array_equal(lfr.to_numpy(lfr.downstream_level(a)), level)
    s = a.topology().stats()
    valid = fd != 255
    assert s["valid_cells"] == valid.sum()
    assert s["ridge_cells"] == (valid & (count == 0)).sum()
    assert s["sink_cells"] == (valid & ~np.isin(fd, list(OFFSETS))).sum()
    assert s["outlet_cells"] == outlets
    assert s["cycle_cells"] == (valid & (level < 0)).sum()
    assert s["max_level"] == max(int(level.max()), 0)
    assert (s["cycle_cells"] > 0) == name.startswith("cycle")
    if s["cycle_cells"] == 0:
        got = lfr.to_numpy(lfr.accu(a, lfr.from_numpy(np.ones(fd.shape, np.float32))))
        assert np.array_equal(got, accu.astype(np.float32), equal_nan=True)


def test_more_tile_rows_than_a_grid_holds(lfr):
    fd = np.full((64 * 65535 + 1, 1), 5, np.uint8)
    with pytest.raises(RuntimeError):
        lfr.from_numpy(fd).topology()
    fd[0], fd[1] = 2, 8  # a cycle: no tiles are needed
    s = lfr.from_numpy(fd).topology().stats()
    assert s["cycle_cells"] == 2 and s["sink_cells"] == fd.size - 2

"""Memory of the path engine: what only the rules with two results use (the cells' positions and the results by position,
12 bytes a cell on large rasters) is there from the first such call on, and not for float64 accu."""
import numpy as np
import pytest

from lue_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lfr():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import framework
    return framework


def _inputs(lfr, shape=(333, 777)):
    rng = np.random.default_rng(11)
    a = lfr.from_numpy(synthetic.flow_direction(*shape, 11, 30.0, wavelength=400))
    m, b = (rng.integers(0, k, shape).astype(np.float32) for k in (4, 12))
    return a, lfr.from_numpy(m), lfr.from_numpy(b), lfr.from_numpy(m.astype(np.float64))


def test_results_by_position_only_where_they_are_used(lfr, monkeypatch):
    monkeypatch.setenv("LUE_GB300_PATH_SPREAD", "0")
    a, m, b, m64 = _inputs(lfr)
    cells = a.shape[0] * a.shape[1]
    device_bytes = lambda: a.topology().stats()["device_bytes"]  # noqa: E731
    lfr.accu(a, m64)
    one = device_bytes()
    first = [lfr.to_numpy(x) for x in lfr.accu_threshold(a, m, b)]
    assert device_bytes() == one + 12 * cells
    for x, y in zip(first, lfr.accu_threshold(a, m, b)):
        assert np.array_equal(x, lfr.to_numpy(y), equal_nan=True)
    assert device_bytes() == one + 12 * cells


def test_first_spread_call_captured(lfr, monkeypatch):
    """The results of a captured first call go straight to the raster (whole numbers: the same bits)."""
    import torch
    monkeypatch.setenv("LUE_GB300_PATH_SPREAD", "0")
    a, m, b, m64 = _inputs(lfr)
    lfr.accu(a, m64)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = lfr.accu_threshold(a, m, b)
    g.replay()
    for x, y in zip(got, lfr.accu_threshold(a, m, b)):
        assert np.array_equal(lfr.to_numpy(x), lfr.to_numpy(y), equal_nan=True)


@pytest.mark.parametrize("what", ["layout", "buffers"])
@pytest.mark.parametrize("op", ["accu", "trigger"])
def test_without_memory_another_engine_does_the_call(lfr, monkeypatch, op, what):
    """Whole numbers: every engine gives the same bits."""
    a, m, b, m64 = _inputs(lfr)
    call = lambda: [lfr.accu(a, m64)] if op == "accu" else list(lfr.accu_trigger(a, m, b))  # noqa: E731
    monkeypatch.setenv("LUE_GB300_PATH_NO_MEMORY", what)
    got = [lfr.to_numpy(x) for x in call()]
    monkeypatch.delenv("LUE_GB300_PATH_NO_MEMORY")
    for x, y in zip(got, call()):
        assert np.array_equal(x, lfr.to_numpy(y), equal_nan=True)


@pytest.mark.parametrize("op", ["accu", "trigger"])
def test_first_call_captured_after_prepare(lfr, op):
    """Whole numbers: a captured first call gives the bits of an ordinary one; so does an ordinary one after it."""
    import torch
    a, m, b, m64 = _inputs(lfr)
    call = lambda: [lfr.accu(a, m64)] if op == "accu" else list(lfr.accu_trigger(a, m, b))  # noqa: E731
    want = [lfr.to_numpy(x) for x in call()]
    first, second = a.topology().clone(), None
    a._topology, second = first, a._topology
    try:
        first.prepare()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = call()
        for _ in range(2):
            g.replay()
        for results in (got, call()):
            for x, w in zip(results, want):
                assert np.array_equal(lfr.to_numpy(x), w, equal_nan=True)
        del g
    finally:
        torch.cuda.synchronize()
        a._topology = second
        first.close()

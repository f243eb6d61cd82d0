"""Path engine calls with infinite material (or thresholds): they are redone along the paths with the walk engine's cell
rules, so the results are that engine's bit for bit; with results spread by position too, and when the redo's own
waits give up and the walk engine does the call.  A trigger that nothing reaches needs no redo.

Tolerance of the last: that of the float32 operations against the float64 oracle."""
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


def _inputs(shape, seed=53):
    fd = synthetic.flow_direction(*shape, seed, 60.0, wavelength=max(shape) / 2).copy()
    rng = np.random.default_rng(seed)
    fd[rng.random(shape) < 0.001] = 255
    m = rng.lognormal(0.0, 1.0, shape)
    m[rng.random(shape) < 0.0005] = np.nan
    return fd, m, rng


def _call(lfr, a, op, m, b):
    if op == "accu":
        return [lfr.to_numpy(lfr.accu(a, lfr.from_numpy(m)))]
    return [lfr.to_numpy(x) for x in getattr(lfr, f"accu_{op}")(a, lfr.from_numpy(m.astype(np.float32)), lfr.from_numpy(b))]


@pytest.mark.parametrize("hook", [None, ("SPREAD", "0"), ("REDO_POLLS", "0")], ids=["default", "results spread", "walk"])
@pytest.mark.parametrize("op", ["accu", "threshold", "fraction", "capacity", "trigger"])
@pytest.mark.parametrize("shape", [(1, 300), (333, 777), (1200, 1501)])
def test_infinite_material(lfr, monkeypatch, shape, op, hook):
    if hook:
        monkeypatch.setenv("LUE_GB300_PATH_" + hook[0], hook[1])
    fd, m, rng = _inputs(shape)
    b = rng.random(shape, dtype=np.float32)
    inf = m.copy()
    inf[shape[0] // 2, shape[1] // 2] = np.inf
    a = lfr.from_numpy(fd)
    normal = _call(lfr, a, op, m, b)
    got = _call(lfr, a, op, inf, b)
    for g, w in zip(_call(lfr, a, op, m, b), normal):  # the call after it is a normal one
        assert np.array_equal(g, w, equal_nan=True)
    monkeypatch.setenv("LUE_GB300_ENGINE", "walk")
    for g, w in zip(got, _call(lfr, a, op, inf, b)):
        assert np.array_equal(g, w, equal_nan=True)


@pytest.mark.parametrize("longest", [None, "0"], ids=["default", "look-back on every level"])
def test_triggers_that_nothing_reaches(lfr, monkeypatch, longest):
    if longest:
        monkeypatch.setenv("LUE_GB300_PATH_FREE_LONGEST", longest)
    fd, m, rng = _inputs((700, 901))
    b = (3.0 * rng.lognormal(0.0, 1.0, fd.shape)).astype(np.float32)
    b[rng.random(fd.shape) < 0.1] = np.inf
    m = m.astype(np.float32)
    want = oracle.accu_trigger(fd, m.astype(np.float64), b.astype(np.float64), fd.shape, dtype=np.float64)
    for g, w, name in zip(_call(lfr, lfr.from_numpy(fd), "trigger", m, b), want, ("outflow", "remainder")):
        parity.assert_close32(g, w, name)

"""Rivers of many scan tiles on the path engine: the tiles before a tile are composed in an order that the layout fixes,
so a repeated call gives the same bits, in plain doubles too, whichever CTA was faster.

Tolerance of the long path's values: a position's sum takes at most 4 (its thread) + 5 + 8 (its CTA) + 6 (its window of 32
tiles) + 31 (the published prefixes of 1000 tiles) additions one after the other, of terms >= 0: below 64 x 2^-53."""
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


def _repeat(lfr, call, runs=20):
    import torch
    first = [x.data.clone() for x in call()]
    for _ in range(runs):
        for x, f in zip(call(), first):
            assert torch.equal(x.data.view(torch.uint8), f.view(torch.uint8))
    return first


@pytest.mark.parametrize("rows, cols", [(1, 256), (3, 600), (40, 821), (997, 1009)])
def test_one_path_through_every_cell(lfr, rows, cols):
    fd = np.full((rows, cols), 6, np.uint8)
    fd[1::2] = 4
    fd[0::2, -1] = 2
    fd[1::2, 0] = 2
    m = np.random.default_rng(rows).lognormal(0.0, 1.0, fd.shape)
    a, x = lfr.from_numpy(fd), lfr.from_numpy(m)
    got = _repeat(lfr, lambda: [lfr.accu(a, x)])[0].cpu().numpy()
    got[1::2], m[1::2] = got[1::2, ::-1].copy(), m[1::2, ::-1].copy()
    want = np.cumsum(m.ravel().astype(np.longdouble)).reshape(m.shape)
    assert np.all(np.abs(got - want) <= 64 * 2.0 ** -53 * want)


@pytest.mark.parametrize("longest", [None, "0"], ids=["default", "look-back on every level"])
@pytest.mark.parametrize("op", ["accu", "trigger", "fraction"])
def test_repeated_calls_give_the_same_bits(lfr, monkeypatch, op, longest):
    if longest:
        monkeypatch.setenv("LUE_GB300_PATH_FREE_LONGEST", longest)
    fd = synthetic.flow_direction(3001, 2777, 41, 200.0, wavelength=3001)
    rng = np.random.default_rng(41)
    a = lfr.from_numpy(fd)
    m = rng.lognormal(0.0, 1.0, fd.shape)
    if op == "accu":
        x = lfr.from_numpy(m)
        _repeat(lfr, lambda: [lfr.accu(a, x)])
        return
    x = lfr.from_numpy(m.astype(np.float32))
    b = lfr.from_numpy(rng.random(fd.shape, dtype=np.float32) * np.float32(1.0 if op == "fraction" else 3.0))
    _repeat(lfr, lambda: getattr(lfr, f"accu_{op}")(a, x, b))


def test_one_path_over_several_prefixes(lfr):
    """4.2 million cells on one path: more than 4000 scan tiles, prefixes published at tiles 1024, 2048, ...; a position's sum
    takes at most 4 + 5 + 8 + 2 x 6 + 1 + 5 additions one after the other."""
    rows, cols = 2100, 2003
    fd = np.full((rows, cols), 6, np.uint8)
    fd[1::2] = 4
    fd[0::2, -1] = 2
    fd[1::2, 0] = 2
    m = np.random.default_rng(3).lognormal(0.0, 1.0, fd.shape)
    a, x = lfr.from_numpy(fd), lfr.from_numpy(m)
    got = _repeat(lfr, lambda: [lfr.accu(a, x)])[0].cpu().numpy()
    got[1::2], m[1::2] = got[1::2, ::-1].copy(), m[1::2, ::-1].copy()
    want = np.cumsum(m.ravel().astype(np.longdouble)).reshape(m.shape)
    assert np.all(np.abs(got - want) <= 64 * 2.0 ** -53 * want)

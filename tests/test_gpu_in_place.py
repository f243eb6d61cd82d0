"""accu (float64) and accu_trigger (float32) through the C interface with an output that is an input: with an infinite cell,
whose call is redone from the inputs on the path engine, the results are those of a call out of place with the
engine that such calls take (bit for bit: the stage engine and the redo both have the walk engine's cell rules)."""
import numpy as np
import pytest

from lue_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(65, 31), (333, 777)])
@pytest.mark.parametrize("op", ["accu", "trigger"])
def test_infinite_material_in_place(op, shape):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lue_gb300 import _lib, framework as lfr
    L = _lib.lib()
    a = lfr.from_numpy(synthetic.flow_direction(*shape, 3, 60.0, wavelength=max(shape) / 2))
    rng = np.random.default_rng(3)
    m = rng.lognormal(0.0, 1.0, shape)
    m[shape[0] // 2, shape[1] // 2] = np.inf
    t = a.topology()
    if op == "accu":
        want = [lfr.accu(a, lfr.from_numpy(m)).data]
        x = torch.from_numpy(m).cuda()
        _lib.check(L.lue_gpu_accu_f64(t.handle, x.data_ptr(), 0.0, x.data_ptr(), None))
        got = [x]
    else:
        b = torch.from_numpy(rng.lognormal(1.0, 1.0, shape).astype(np.float32)).cuda()
        x = torch.from_numpy(m.astype(np.float32)).cuda()
        want = [y.data for y in lfr.accu_trigger(a, lfr.PartitionedArray(x.clone()), lfr.PartitionedArray(b.clone()))]
        _lib.check(L.lue_gpu_accu_trigger_f32(t.handle, x.data_ptr(), 0.0, b.data_ptr(), 0.0, x.data_ptr(), b.data_ptr(), None))
        got = [x, b]
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w.cpu().numpy(), equal_nan=True)

"""wb_find_blocks and wb_points_in into arrays on the device and in pinned host
memory: the same answers as into an ordinary host array."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["device", "pinned"])
@pytest.mark.parametrize("r", [0.3, 2.0, 1e6])
def test_answers_into_device_memory(classifier, where, r):
    from wolkenbase_gb300 import synth
    cloud = synth.density_tile(30000, 84)
    classifier.build(cloud)
    d = cloud.decoded()
    v = tuple(d[:, :2].mean(axis=0))
    sh = classifier._shape(1, v, r, 1.0)

    def buf(n, dtype):
        return torch.full((n,), -1, dtype=dtype, device="cuda") if where == "device" else \
            torch.full((n,), -1, dtype=dtype).pin_memory()

    n = C.c_uint64(0)
    want = classifier.find_blocks(1, v, r)
    out = buf(want.size + 3, torch.int64)
    assert classifier.L.wb_find_blocks(classifier.ctx, C.byref(sh), C.c_void_p(out.data_ptr()), out.numel(), C.byref(n)) == 0
    got = out.cpu().numpy()
    assert n.value == want.size and np.array_equal(got[:want.size], want) and np.all(got[want.size:] == -1)
    for srt in (0, 1):
        want = classifier.points_in(1, v, r, sorted=bool(srt))
        out = buf(want.size + 3, torch.int32)
        assert classifier.L.wb_points_in(classifier.ctx, C.byref(sh), srt, C.c_void_p(out.data_ptr()), out.numel(), C.byref(n)) == 0
        got = out.cpu().numpy()
        assert n.value == want.size and np.array_equal(got[:want.size].view(np.uint32), want)
        assert np.all(got[want.size:] == -1)

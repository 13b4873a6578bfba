"""Host outputs of a frame, through the pinned buffer (small frames) and by direct copies:
both planes, one plane, and pipelined frames give the device outputs' bytes."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
from briefmatch_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("W,H", [(40, 24), (128, 96), (129, 96), (160, 120)])   # 12288 pixels is the line
@pytest.mark.parametrize("pipelined", [False, True])
def test_host_equals_device_output(W, H, pipelined):
    prm = bm.BMParams.derive(W, H, 1.5, 1.5, N=64)
    frames, _ = synth.make_sequence(5, W, H, 3, vmax=3.0)
    eng = bm.BriefMatch(prm)
    eng.setup()
    eng.set_pipelined(pipelined)
    dev = torch.empty(2, 2, H, W, device="cuda")
    host = np.full((2, 2, H, W), np.nan, np.float32)
    only_v = np.full((2, H, W), np.nan, np.float32)
    conv = []
    for mode in ("device", "host", "v"):
        eng.reset_sequence()
        eng.set_rng_position(0)
        eng.frame(frames[0].ctypes.data, False)
        for k in (1, 2):
            if mode == "device":
                eng.frame(frames[k].ctypes.data, False, dev[k - 1, 0].data_ptr(), dev[k - 1, 1].data_ptr(), True)
                conv.append([np.asarray(a).reshape(H, W).copy() for a in eng.convert()])
            elif mode == "host":
                eng.frame(frames[k].ctypes.data, False, host[k - 1, 0].ctypes.data, host[k - 1, 1].ctypes.data, False)
            else:
                eng.frame(frames[k].ctypes.data, False, None, only_v[k - 1].ctypes.data, False)
            eng.synchronize()
    want = dev.cpu().numpy()
    assert np.array_equal(host, want)
    assert np.array_equal(only_v, want[:, 1])
    assert np.array_equal(np.asarray(conv), want)

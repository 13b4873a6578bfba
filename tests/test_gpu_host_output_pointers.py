"""Outputs asked for as host memory but handed over as device memory: the copies follow the
pointer whatever the frame's size, through the host buffer of small frames and without."""
from __future__ import annotations

import ctypes
import time

import numpy as np
import pytest

import briefmatch_gb300 as bm
from briefmatch_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("W,H", [(40, 24), (96, 64), (160, 120)])
def test_device_memory_as_host_output(W, H):
    prm = bm.BMParams.derive(W, H, 1.5, 1.5, N=64)
    frames = synth.make_pair(5, W, H, 3.0)[:2]
    eng = bm.FlowEngine(prm)
    eng.process_frame(frames[0])
    want = eng.process_frame(frames[1])
    dev = torch.zeros(2, 2, H, W, device="cuda")
    host = np.zeros((H, W), np.float32)
    torch.cuda.synchronize()
    eng.reset_sequence()
    eng.set_rng_position(0)
    eng.process_frame(frames[0])
    eng.frame(frames[1].ctypes.data, False, dev[0, 0].data_ptr(), dev[0, 1].data_ptr(), False)
    eng.synchronize()
    bm.check(bm.lib().bm_convert(eng.ctx, ctypes.c_void_p(host.ctypes.data), ctypes.c_void_p(dev[1, 1].data_ptr())))
    eng.synchronize()
    got = dev.cpu().numpy()
    assert np.array_equal(got[0, 0], want[0]) and np.array_equal(got[0, 1], want[1])
    assert np.array_equal(host, want[0]) and np.array_equal(got[1, 1], want[1])
    eng.clean()


def test_a_small_context_is_made_as_fast_as_a_larger_one():
    """Contexts with the host buffer (96x64) and without it (160x120), in turn: the smaller
    one's buffers are made and freed in less time, page-locked memory would double it."""
    params = [bm.BMParams.derive(W, H, 1.5, 1.5, N=64) for W, H in ((96, 64), (160, 120))]
    times = ([], [])
    for _ in range(25):
        for prm, t in zip(params, times):
            t0 = time.perf_counter()
            eng = bm.BriefMatch(prm)
            eng.setup()
            eng.clean()
            t.append(time.perf_counter() - t0)
    small, large = (float(np.median(t)) for t in times)
    assert small <= 1.2 * large

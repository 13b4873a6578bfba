"""Chained launches of a frame (each may start under the last blocks of the one before):
the flow of bm_frame equals, bit for bit and every time, the same stages called one by one
with a synchronisation after each, on grids from a few blocks (where two launches share the
SMs throughout) to several waves, with and without resampling."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
from bmtest import make_engine, random_image, small_params

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("W,H,u,N", [(33, 9, 2.0, 64), (96, 64, 1.5, 128), (200, 121, 1.0, 128), (320, 240, 2.9, 512),
                                     (640, 361, 2.9, 32)])
def test_frame_equals_synchronised_stages(W, H, u, N):
    prm = small_params(W, H, u, u, N=N)
    eng, _ = make_engine(prm)
    rng = np.random.default_rng(W)
    base = random_image(rng, W + 8, H + 8)
    f = [np.clip(base[k:k + H, 2 * k:2 * k + W], 0, 255).astype(np.uint8) for k in (0, 3)]
    d8 = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in f]
    d32 = [a.float() for a in d8]
    up = [torch.empty(prm.sy, prm.sx, device="cuda") for _ in range(2)]
    sync = torch.cuda.synchronize
    sync()
    for k in range(2):
        if u == 1.0:
            up[k].copy_(d32[k])
        else:
            eng.upsample(d32[k].data_ptr(), up[k].data_ptr())
        sync()
        eng.features(up[k].data_ptr(), k)
        sync()
    eng.set_rng_position(0)
    eng.initialize(True)
    sync()
    pd = -1
    for _ in range(prm.iterations):
        eng.propagate(pd)
        sync()
        eng.random_search()
        sync()
        pd = -pd
    eng.downsample()
    sync()
    eng.process(d32[0].data_ptr())
    sync()
    want = eng.read_buffer(bm.BM_BUF_FLOW_OUT, np.float32).reshape(2, H, W)
    got = torch.empty(10, 2, H, W, device="cuda")
    for r in range(got.shape[0]):
        eng.reset_sequence()
        eng.set_rng_position(0)
        eng.frame(d8[0].data_ptr(), True)
        eng.frame(d8[1].data_ptr(), True, got[r, 0].data_ptr(), got[r, 1].data_ptr(), True)
    sync()
    for r in range(got.shape[0]):
        assert np.array_equal(got[r].cpu().numpy(), want), r

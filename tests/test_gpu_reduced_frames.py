"""Frames reduced by re-sampling (factors below 1, on either side of the line where output
rows stop sharing windows): image, float frame, descriptors and flow of bm_frame equal the
stage-by-stage calls', and a batch's flow equals bm_frame's."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
from briefmatch_gb300 import synth
from bmtest import engine_features, make_engine, small_params

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("W,H,ux,uy", [(211, 143, 0.1, 0.1), (230, 140, 0.13, 0.13), (230, 140, 0.13, 0.15),
                                       (150, 121, 0.5, 0.5), (64, 203, 2.0, 0.11), (300, 40, 0.1, 1.7)])
def test_reduced_frames(W, H, ux, uy):
    prm = small_params(W, H, ux, uy, N=64)
    frames = synth.make_pair(3, W, H, 3.0)[:2]
    eng, pattern = make_engine(prm)
    d = [torch.from_numpy(f).cuda() for f in frames]
    ups = [torch.empty(prm.sy, prm.sx, device="cuda") for _ in d]
    torch.cuda.synchronize()
    want = []
    for k in range(2):
        eng.upsample_u8(d[k].data_ptr(), ups[k].data_ptr())
        eng.features(ups[k].data_ptr(), k)
        torch.cuda.synchronize()
        want.append(engine_features(eng, k))
    got = bm.FlowEngine(prm)
    got.set_pattern(pattern)
    for k in range(2):
        u, v = got.process_frame(frames[k])
        up = got.read_buffer(bm.BM_BUF_UP, np.float32, prm.sx * prm.sy).reshape(prm.sy, prm.sx)
        frame = got.read_buffer(bm.BM_BUF_FRAME_PREV, np.float32, W * H).reshape(H, W)
        assert np.array_equal(up, ups[k].cpu().numpy())
        assert np.array_equal(frame, frames[k].astype(np.float32))
        assert np.array_equal(engine_features(got, 0), want[k])
    b = bm.Batch([prm])
    b.set_pattern(0, pattern)
    b.set_schedule(per_pair=1)
    b.load_frames(b.pack_frames([frames]))
    b.run()
    b.synchronize()
    (bu, bv), = b.read_flows()
    b.close()
    assert np.array_equal(bu, u) and np.array_equal(bv, v)

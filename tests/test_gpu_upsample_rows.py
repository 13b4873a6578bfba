"""Up-sampling of a frame with every number of rows per thread (chosen by the grid's size),
odd heights so that the last thread's rows are cut: image, descriptors and float frame
equal, bit for bit, those of the stage-by-stage calls (one output per thread)."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
from bmtest import engine_features, make_engine, random_image, small_params

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("W,H,u", [(61, 41, 2.0), (203, 131, 2.0), (301, 191, 2.0), (437, 251, 2.0), (150, 91, 4.9),
                                   (320, 203, 1.1)])
def test_rows_per_thread(W, H, u):
    prm = small_params(W, H, u, u, N=64)
    eng, _ = make_engine(prm)
    img = np.clip(random_image(np.random.default_rng(W), W, H), 0, 255).astype(np.uint8)
    d = torch.from_numpy(img).cuda()
    ref = torch.empty(prm.sy, prm.sx, device="cuda")
    torch.cuda.synchronize()
    eng.upsample_u8(d.data_ptr(), ref.data_ptr())
    eng.features(ref.data_ptr(), 0)
    torch.cuda.synchronize()
    want = engine_features(eng, 0)
    got = bm.BriefMatch(prm)
    got.setup()
    got.set_pattern(prm.make_pattern(3))
    got.frame(d.data_ptr(), True)
    got.synchronize()
    up = got.read_buffer(bm.BM_BUF_UP, np.float32, prm.sx * prm.sy).reshape(prm.sy, prm.sx)
    assert np.array_equal(up, ref.cpu().numpy())
    assert np.array_equal(engine_features(got, 0), want)

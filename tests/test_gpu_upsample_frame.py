"""The float frame that the up-sampling writes beside its image, for every number of rows per
thread (chosen by the grid's size) and frames with more and fewer pixels than its threads:
the 8-bit frame's values."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("W,H,u,rows", [(61, 41, 2.0, 2), (203, 131, 2.0, 2), (270, 201, 2.0, 4), (550, 300, 2.0, 8),
                                        (320, 203, 1.1, 2), (901, 811, 0.2, 2), (1000, 901, 0.5, 4), (1500, 1403, 0.5, 8)])
def test_float_frame(W, H, u, rows):
    prm = bm.BMParams.derive(W, H, u, u, N=64)
    pattern = prm.make_pattern(3)
    m = int(np.abs(pattern.astype(np.int64)).max())
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = -(-(prm.sx + 2 * m) // 32) * -(-(prm.sy + 2 * m) // 8)
    assert rows == (8 if tiles >= 8 * sms else 4 if tiles >= 4 * sms else 2)
    img = np.random.default_rng(W).integers(0, 256, (H, W), dtype=np.uint8)
    eng = bm.FlowEngine(prm)
    eng.set_pattern(pattern)
    for k in range(2):
        eng.process_frame(img if k == 0 else img[::-1])
        got = eng.read_buffer(bm.BM_BUF_FRAME_PREV, np.float32, W * H).reshape(H, W)
        assert np.array_equal(got, (img if k == 0 else img[::-1]).astype(np.float32))
    eng.clean()

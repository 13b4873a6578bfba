"""Descriptors of frames flat in part: warps that leave the keys for the float image at a
chunk's first samples, in the middle of a chunk, and not at all, next to each other."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
import oracle
from bmtest import engine_features, random_image

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


def _image(kind, rng, w, h):
    img = np.clip(np.rint(random_image(rng, w, h)), 0, 255).astype(np.uint8)
    if kind == "letterbox":
        img[:h // 3] = 0
        img[-h // 4:] = 16
    elif kind == "left":
        img[:, :w // 2] = 255
    elif kind == "spots":        # some samples of every pixel tie
        img[rng.random((h, w)) < 0.6] = 128
    return img


@pytest.mark.parametrize("kind", ["letterbox", "left", "spots"])
@pytest.mark.parametrize("W,H,u,N", [(70, 45, 2.9, 32), (45, 23, 1.5, 50), (64, 33, 2.0, 128), (41, 40, 3.3, 200),
                                     (52, 18, 4.9, 512)])
def test_partly_flat_frames(kind, W, H, u, N):
    prm = bm.BMParams.derive(W, H, u, u, N=N, patch_radius=5.0)
    eng = bm.BriefMatch(prm)
    eng.setup()
    pattern = prm.make_pattern(8)
    pattern[8:12] = 0.0          # a sample whose two points coincide, among the first eight
    eng.set_pattern(pattern)
    d = torch.from_numpy(_image(kind, np.random.default_rng(W), W, H)).cuda()
    torch.cuda.synchronize()
    eng.frame(d.data_ptr(), True)
    eng.synchronize()
    up = eng.read_buffer(bm.BM_BUF_UP, np.float32, prm.sx * prm.sy).reshape(prm.sy, prm.sx)
    assert np.array_equal(engine_features(eng, 0), oracle.features(up, pattern, N))

"""Frame descriptors decided on 16-bit keys, bit for bit against the oracle on the
engine's up-sampled image: textures, images where most samples are equal, images whose
Lanczos overshoot leaves the keys' range, odd sizes and every descriptor length."""
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
    if kind == "texture":
        return np.clip(np.rint(random_image(rng, w, h)), 0, 255).astype(np.uint8)
    if kind == "flat":      # one grey level and a few other pixels: nearly every pair ties
        img = np.full((h, w), 200, np.uint8)
        img[rng.random((h, w)) < 0.02] = 13
        return img
    if kind == "binary":    # 0 / 255 noise: overshoot beyond both ends of the key range
        return (rng.integers(0, 2, (h, w)) * 255).astype(np.uint8)
    ramp = np.linspace(0, 255, w)[None, :].repeat(h, 0)   # neighbours closer than a key step
    return np.rint(ramp / 16).astype(np.uint8)


@pytest.mark.parametrize("kind", ["texture", "flat", "binary", "ramp"])
@pytest.mark.parametrize("W,H,u,N", [(44, 31, 2.9, 128), (45, 23, 1.5, 31), (64, 33, 2.0, 64), (23, 40, 3.3, 250),
                                     (32, 18, 4.9, 512)])
def test_frame_descriptors(kind, W, H, u, N):
    prm = bm.BMParams.derive(W, H, u, u, N=N, patch_radius=8.0)
    eng = bm.BriefMatch(prm)
    eng.setup()
    pattern = prm.make_pattern(5)
    pattern[4:8] = 0.0           # a sample whose two points coincide
    eng.set_pattern(pattern)
    img = _image(kind, np.random.default_rng(W), W, H)
    d = torch.from_numpy(img).cuda()
    torch.cuda.synchronize()
    eng.frame(d.data_ptr(), True)
    eng.synchronize()
    up = eng.read_buffer(bm.BM_BUF_UP, np.float32, prm.sx * prm.sy).reshape(prm.sy, prm.sx)
    assert np.array_equal(engine_features(eng, 0), oracle.features(up, pattern, N))

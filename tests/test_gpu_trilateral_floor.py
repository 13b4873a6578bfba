"""Outputs whose weights sum to less than the filter's floor of 1e-5: there the weights
themselves count, not their quotients, and their exponents are large."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
import oracle
from bmtest import random_image, trilateral_f64

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("W,H,sS", [(96, 64, 0.3), (200, 64, 0.7), (97, 61, 1.1), (1024, 330, 0.7), (70, 66, 1.5)])
@pytest.mark.parametrize("speed", [18.0, 90.0, 700.0])
def test_sums_under_the_floor(W, H, sS, speed):
    """Rough fields, whose medians lie between their samples, and a narrow range: most sums of
    weights are small.  The flow changes its sign every 16 columns, so that half of the
    outputs are far from any one flow.  A weight's relative error is its exponent's absolute one times ln 2;
    the exponents that count are below 27, their three terms' differences, squares and sums
    rounded to 2^-24 of themselves (six at most), and the intensity's scaled centre (up to 8.5,
    differences up to 4) adds 2^-18: 2^-16 in all, of an output that is below the floor's
    share of the flow."""
    rng = np.random.default_rng(int(W + speed))
    sign = np.where(np.arange(W) // 16 % 2, 1.0, -1.0)
    U, V = ((speed * sign + rng.uniform(-2, 2, (H, W))).astype(np.float32) for _ in range(2))
    I = random_image(rng, W, H)
    d = [torch.from_numpy(a).cuda() for a in (U, V, np.ascontiguousarray(I, np.float32))]
    out = torch.empty(2, H, W, device="cuda")
    torch.cuda.synchronize()
    bm.refine_noalloc(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), W, H, 3,
                      0.1, 0.1, sS)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    Um, Vm = (oracle.median1d(oracle.median1d(a, 1, 3), 0, 3) for a in (U, V))
    s = int(np.ceil(2.5 * float(np.float32(sS))))
    under = 0
    for r0 in (0, H // 2, H - 8):
        e = np.stack(trilateral_f64(U, V, Um, Vm, I, r0, 8, s, 0.1, 0.1, sS))
        low = (np.abs(e[0]) > 1e-3 * speed) & (np.abs(e[0]) < 0.5 * speed)   # the sum of weights is below the floor
        under += int(low.sum())
        off = np.abs(got[:, r0:r0 + 8] - e)
        assert (off <= 2.0 ** -16 * np.abs(e))[:, low].all(), (off / np.abs(e))[:, low].max()
    assert under >= 20

"""The cross-trilateral filter against float64 over its block shapes (thread rows chosen
by tile count and window), window parities, frames smaller than a tile or than the
window, and fields with unknown (huge, infinite, NaN) vectors."""
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

FLOW_TOL = 1e-4      # refined flow, px max-abs: the bar of every refinement test


def _refine(U, V, I, fsize, sEPE, sI, sS):
    H, W = U.shape
    d = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (U, V, I)]
    out = torch.empty(2, H, W, device="cuda")
    torch.cuda.synchronize()
    bm.refine_noalloc(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), W, H,
                      fsize, sEPE, sI, sS)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _field(rng, W, H):
    U = rng.normal(0, 0.6, (H, W)) + np.linspace(-20, 20, W)[None, :]
    U[:, W // 2:] += 15.0        # a motion edge
    return U.astype(np.float32), rng.normal(3, 0.6, (H, W)).astype(np.float32)


# sS -> half window ceil(2.5 sS); the last three frames are past two tiles per SM
@pytest.mark.parametrize("W,H,sS", [(40, 30, 0.3), (33, 65, 0.8), (5, 9, 1.1), (100, 37, 2.0), (64, 64, 8.4),
                                    (95, 50, 9.2), (130, 140, 13.0), (97, 71, 20.8), (1024, 320, 0.4),
                                    (1000, 333, 3.1), (1600, 220, 6.0)])
def test_block_shapes_and_windows(W, H, sS):
    rng = np.random.default_rng(W + H)
    U, V = _field(rng, W, H)
    I = random_image(rng, W, H)
    out = _refine(U, V, I, 3, 0.4, 0.1, sS)
    Um, Vm = (oracle.median1d(oracle.median1d(a, 1, 3), 0, 3) for a in (U, V))
    s = int(np.ceil(2.5 * float(np.float32(sS))))   # 2.5 * sqrt(sS^2) in double, briefmatch_cuda.cu:266
    for r0 in sorted({0, max(0, H // 2 - 1), max(0, H - 3)}):
        rows = min(3, H - r0)
        eu, ev = trilateral_f64(U, V, Um, Vm, I, r0, rows, s, 0.4, 0.1, sS)
        assert np.abs(out[0, r0:r0 + rows] - eu).max() <= FLOW_TOL
        assert np.abs(out[1, r0:r0 + rows] - ev).max() <= FLOW_TOL


@pytest.mark.parametrize("bad", [1e10, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("W,H", [(96, 72), (1024, 330)])
def test_unknown_vectors_stay_local(bad, W, H):
    """A bad vector reaches the outputs whose windows hold it and no others."""
    rng = np.random.default_rng(W)
    U, V = _field(rng, W, H)
    I = random_image(rng, W, H)
    s = 5
    clean = _refine(U, V, I, 1, 0.4, 0.1, 2.0)
    spoilt = U.copy()
    y, x = H // 2 + 1, W // 2 + 3
    spoilt[y, x] = bad
    out = _refine(spoilt, V, I, 1, 0.4, 0.1, 2.0)
    yy, xx = np.mgrid[0:H, 0:W]
    # output p reads q in [p - s, p + s): it holds (x, y) when x - s < px <= x + s
    far = (xx <= x - s) | (xx > x + s) | (yy <= y - s) | (yy > y + s)
    assert np.isfinite(clean).all()
    # a block takes its samples relative to one of its medians: with another one the
    # roundings differ (flows to 40 px: 1e-5 is four units in the last place)
    assert np.abs(out[0] - clean[0])[far].max() <= 1e-5 and np.abs(out[1] - clean[1])[far].max() <= 1e-5
    assert np.isfinite(out[:, far]).all()
    if np.isfinite(bad):
        assert np.isfinite(out).all()

"""The cross-trilateral filter's value depends on its window alone and is as fine as its own
flow: small flows beside a fast object, changes outside the window, and centres near and
past the largest float."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
from bmtest import random_image, trilateral_f64

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


def _refine(U, V, I, sS, sE=0.4):
    H, W = U.shape
    d = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (U, V, I)]
    out = torch.empty(2, H, W, device="cuda")
    torch.cuda.synchronize()
    bm.refine_noalloc(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), W, H,
                      1, sE, 0.1, sS)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _half_window(sS):
    return int(np.ceil(2.5 * float(np.float32(sS))))   # in double, of the float (briefmatch_cuda.cu:266)


def _bad(W, H, reach=0):
    """Pixels at and around the middles of the blocks of every height (8, 16 and 32 rows)."""
    yy, xx = np.mgrid[0:H, 0:W]
    return (np.abs(xx % 32 - 16) <= reach) & ((yy % 8 == 4) | (yy % 16 == 8) | (yy % 32 == 16))


# one, and many, 32x32 tiles per SM; window 2s
@pytest.mark.parametrize("W,H,sS", [(96, 72, 6.0), (1024, 352, 3.2), (160, 96, 18.8)])
@pytest.mark.parametrize("speed", [3.0, 60.0, 1000.0])
def test_small_flow_beside_a_fast_object(W, H, sS, speed):
    """Background outputs are held to the background's own size: half a unit in the last
    place for the sum centre + quotient (2^-24), and the summed differences' errors -- each
    weight's 2^-20 from the rounding of an exponent below 16 and the exponential's own error,
    up to 52 roundings of 2^-24 along a column -- on differences of at most 0.02 px: 2^-19 of
    that in all.  The object's weights, below 2^-40, count for nothing."""
    rng = np.random.default_rng(W)
    obj = _bad(W, H, 2)
    U, V = (np.where(obj, k * speed, 0.01 + rng.uniform(-0.005, 0.005, (H, W))).astype(np.float32) for k in (1, -1))
    I = random_image(rng, W, H)
    out = _refine(U, V, I, sS)
    s = _half_window(sS)
    for r0 in (0, H // 2, H - 2):
        eu, ev = trilateral_f64(U, V, U, V, I, r0, 2, s, 0.4, 0.1, sS)
        back = ~obj[r0:r0 + 2]
        assert np.abs(out[0, r0:r0 + 2] - eu)[back].max() <= 2.0 ** -19 * 0.02
        assert np.abs(out[1, r0:r0 + 2] - ev)[back].max() <= 2.0 ** -19 * 0.02


@pytest.mark.parametrize("W,H", [(96, 72), (1024, 330)])
@pytest.mark.parametrize("bad", [700.0, 1e10, np.inf, np.nan])
def test_nothing_outside_the_window_counts(W, H, bad):
    rng = np.random.default_rng(W)
    U = (rng.normal(0, 0.6, (H, W)) + np.linspace(-20, 20, W)[None, :]).astype(np.float32)
    V = rng.normal(3, 0.6, (H, W)).astype(np.float32)
    I = random_image(rng, W, H)
    s = _half_window(1.2)
    clean = _refine(U, V, I, 1.2)
    spoilt, far = U.copy(), np.ones((H, W), bool)
    yy, xx = np.mgrid[0:H, 0:W]
    for y, x in zip(*np.nonzero(_bad(W, H) & (yy // 32 % 2 == 0) & (xx // 32 % 2 == 0))):
        spoilt[y, x] = bad
        # output p reads q in [p - s, p + s)
        far &= (xx <= x - s) | (xx > x + s) | (yy <= y - s) | (yy > y + s)
    out = _refine(spoilt, V, I, 1.2)
    assert far.any() and not far.all()
    assert np.array_equal(out[:, far], clean[:, far])


@pytest.mark.parametrize("bad", [1e20, 2e30, 1e36, 1.5e38, np.inf, -np.inf, np.nan])
def test_far_centres(bad):
    """A far vector has weight 0 in its neighbours' windows and weight 1, alone, in its own;
    an infinite or NaN one makes its plane NaN wherever a window holds it."""
    W, H, s = 64, 48, _half_window(1.6)
    rng = np.random.default_rng(4)
    U = rng.normal(2, 0.1, (H, W)).astype(np.float32)
    V = rng.normal(3, 0.1, (H, W)).astype(np.float32)
    I = random_image(rng, W, H)
    clean = _refine(U, V, I, 1.6)
    y, x = 21, 30
    U[y, x] = bad
    out = _refine(U, V, I, 1.6)
    yy, xx = np.mgrid[0:H, 0:W]
    near = (xx > x - s) & (xx <= x + s) & (yy > y - s) & (yy <= y + s)
    own = (xx == x) & (yy == y)
    assert np.array_equal(out[:, ~near], clean[:, ~near])
    if np.isfinite(bad):
        assert np.abs(out[0, y, x] - bad) <= 1e-6 * bad and np.abs(out[1, y, x] - V[y, x]) <= 1e-6
        assert np.abs(out - clean)[:, near & ~own].max() <= 1.0 and np.isfinite(out).all()
    else:
        assert np.isnan(out[0][near]).all() and np.isnan(out[1, y, x])


@pytest.mark.parametrize("sS", [0.3, 0.7, 1.1, 1.9, 3.1, 3.5, 6.3])   # half windows 1 to 16
def test_block_shapes_agree(sS):
    """A crop's outputs, whose windows lie inside it, are those of the large frame: blocks of
    8, 16 and 32 rows, one and two groups of columns.  (Crops start at a multiple of the four
    rows a thread owns: which rows of a window pair up follows the row's number.)"""
    rng = np.random.default_rng(11)
    W, H, w, h = 1024, 352, 96, 72
    U = (rng.normal(0, 0.4, (H, W)) + np.linspace(-9, 9, W)[None, :]).astype(np.float32)
    V = rng.normal(3, 0.4, (H, W)).astype(np.float32)
    I = random_image(rng, W, H)
    s = _half_window(sS)
    big = _refine(U, V, I, sS)
    for x0, y0 in ((101, 64), (700, 132)):
        part = _refine(*(a[y0:y0 + h, x0:x0 + w] for a in (U, V, I)), sS)
        inner = (slice(None), slice(s, h - s), slice(s, w - s))
        assert np.array_equal(part[inner], big[:, y0:y0 + h, x0:x0 + w][inner])
    for r0 in (0, 171, H - 2):
        eu, ev = trilateral_f64(U, V, U, V, I, r0, 2, s, 0.4, 0.1, sS)
        assert np.abs(big[0, r0:r0 + 2] - eu).max() <= 1e-5 and np.abs(big[1, r0:r0 + 2] - ev).max() <= 1e-5


def test_window_without_a_tile():
    """Half windows past the largest tile: small flows beside fast ones, and far centres."""
    W, H, sS = 150, 110, 21.5
    rng = np.random.default_rng(5)
    obj = _bad(W, H, 2)
    U = np.where(obj, 500.0, 0.01 + rng.uniform(-0.005, 0.005, (H, W))).astype(np.float32)
    V = np.where(obj, -40.0, 0.01 + rng.uniform(-0.005, 0.005, (H, W))).astype(np.float32)
    I = random_image(rng, W, H)
    s = _half_window(sS)
    assert s > 52
    out = _refine(U, V, I, sS)
    eu, ev = trilateral_f64(U, V, U, V, I, 54, 3, s, 0.4, 0.1, sS)
    back = ~obj[54:57]
    # the sums run over the whole window, 11,000 taps one after the other: 2^-24 each at worst
    tol = 2.0 ** -24 * 0.02 + 11000 * 2.0 ** -24 * 0.01
    assert np.abs(out[0, 54:57] - eu)[back].max() <= tol and np.abs(out[1, 54:57] - ev)[back].max() <= tol
    U[55, 70] = 2e38
    out = _refine(U, V, I, sS)
    assert out[0, 55, 70] == np.float32(2e38) and np.isfinite(out).all()


def test_empty_window():
    """A spatial sigma whose square underflows leaves no taps: every sum is 0, and so is the
    quotient with the floor of the weights, also at NaN and infinite centres."""
    rng = np.random.default_rng(6)
    U, V = (rng.normal(0, 3, (20, 35)).astype(np.float32) for _ in range(2))
    U[3, 4], V[5, 6], U[7, 8] = np.nan, np.inf, 1e35
    assert not _refine(U, V, random_image(rng, 35, 20), 1e-30).any()

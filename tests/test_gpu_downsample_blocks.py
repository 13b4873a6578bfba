"""Block down-sampling by 32, 16 and 8 rows, by the per-pixel form where 8 rows do not fit,
and on either side of the tap count and block count that its use asks for, against the
oracle, bit for bit.  Each case states the form it is there for."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
import oracle
from bmtest import make_engine, random_field, set_field, small_params

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


def _form(prm, taps):
    """Rows per block, or 0 for the per-pixel form: windows of 16 taps and more whose source
    rows (8 bytes a column of 32) fit 48 KB, where blocks of 32 rows give every SM two."""
    def fits(rows):
        return ((rows - 1) * prm.sy // prm.sy_in + 2 + taps) * 32 * 8 <= 48 * 1024

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = -(-prm.sx_in // 32) * -(-prm.sy_in // 32)
    rows = next((r for r in (32, 16, 8) if fits(r)), 0)
    return rows if taps >= 16 and blocks >= 2 * sms else 0


@pytest.mark.parametrize("W,H,uy,sigma,taps,form", [
    (1024, 331, 5.4, 2.6, 17, 32), (1030, 331, 5.7, 2.6, 17, 16), (1024, 331, 11.5, 2.6, 17, 16),
    (1024, 331, 11.8, 2.6, 17, 8), (1017, 347, 14.0, 3.3, 21, 8), (1024, 331, 24.7, 2.6, 17, 8),
    (1024, 331, 25.3, 2.6, 17, 0), (1024, 331, 5.4, 2.3, 15, 0), (1024, 281, 5.4, 2.6, 17, 0)])
def test_rows_per_block(W, H, uy, sigma, taps, form):
    prm = small_params(W, H, 1.0, uy, N=32)
    prm.sigma = sigma
    eng, _ = make_engine(prm)
    got_taps = prm.gauss_taps()
    assert len(got_taps) == taps and _form(prm, taps) == form
    rng = np.random.default_rng(H)
    NX, NY = random_field(rng, prm.sx, prm.sy, 20)
    set_field(eng, NX, NY, np.zeros(prm.sx * prm.sy, np.uint16))
    eng.downsample()
    torch.cuda.synchronize()
    uv = eng.read_buffer(bm.BM_BUF_FLOW_IN, np.float32).reshape(2, H, W)
    U, V = oracle.downsample(NX, NY, prm.sx, prm.sy, W, H, got_taps, eng.nn_indices())
    assert np.array_equal(uv[0], U) and np.array_equal(uv[1], V)

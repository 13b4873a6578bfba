"""Down-sampling by blocks that form each row's horizontal sum once, and per pixel: every
number of rows per block, ragged last blocks, small frames, and a scale whose window does
not fit, against the oracle, bit for bit."""
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


@pytest.mark.parametrize("W,H,u", [(1700, 620, 5.6), (1024, 311, 11.0), (1030, 321, 4.1), (97, 61, 4.9), (33, 20, 24.0),
                                   (5, 3, 2.0)])
def test_downsample_blocks(W, H, u):
    prm = small_params(W, H, u, u, N=32)
    eng, _ = make_engine(prm)
    rng = np.random.default_rng(W + H)
    NX, NY = random_field(rng, prm.sx, prm.sy, 20)
    set_field(eng, NX, NY, np.zeros(prm.sx * prm.sy, np.uint16))
    eng.downsample()
    torch.cuda.synchronize()
    uv = eng.read_buffer(bm.BM_BUF_FLOW_IN, np.float32).reshape(2, H, W)
    U, V = oracle.downsample(NX, NY, prm.sx, prm.sy, W, H, prm.gauss_taps(), eng.nn_indices())
    assert np.array_equal(uv[0], U) and np.array_equal(uv[1], V)

"""Jump-flood levels for every descriptor length's kernel (one thread per descriptor up
to 16 bytes, two or four lanes per longer descriptor) against the oracle, bit for bit:
rows that do not fill the last warp, fields with repeated vectors, steps wider than the
image, and the random search fused into the last level."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
import oracle
from bmtest import engine_features, engine_field, engine_normals, hamming_at, make_engine, random_field, random_image, set_field

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("N", [32, 64, 128, 200, 512])
@pytest.mark.parametrize("sx,sy,jf,double_prop,pd", [(96, 41, 256, 1, -1), (97, 30, 3, 1, 1), (127, 17, 64, 0, -1),
                                                     (33, 65, 1 << 20, 1, 1), (5, 9, 4, 1, -1)])
def test_levels_and_fused_search(N, sx, sy, jf, double_prop, pd):
    prm = bm.BMParams(sx=sx, sy=sy, sx_in=sx, sy_in=sy, N=N, jfMax=jf, doubleProp=double_prop, iterations=2,
                      patchArea=9.0, fsize=3, sS=1.0)
    eng, pattern = make_engine(prm)
    rng = np.random.default_rng(N + sx)
    ups = [torch.from_numpy(random_image(rng, sx, sy)).cuda() for _ in range(2)]
    torch.cuda.synchronize()
    for slot in (0, 1):
        eng.features(ups[slot].data_ptr(), slot)
    F1, F2 = engine_features(eng, 0), engine_features(eng, 1)
    NX0, NY0 = random_field(rng, sx, sy, 6)
    coarse = rng.random(NX0.shape) < 0.5  # half the field repeats vectors, so candidates coincide
    NX0, NY0 = np.where(coarse, 0, NX0), np.where(coarse, 0, NY0)
    H0 = hamming_at(F1, F2, sx, NX0, NY0)
    set_field(eng, NX0, NY0, H0)
    eng.propagate(pd)
    nx, ny, cost, _ = engine_field(eng)
    NX, NY, H = oracle.propagate(F1, F2, sx, sy, N, pd, jf, double_prop, NX0, NY0, H0)
    assert np.array_equal(nx, NX) and np.array_equal(ny, NY) and np.array_equal(cost, H)
    # the whole match: initialisation, then two passes with the search in their last level
    normals = [engine_normals(eng, c) for c in range(2)]
    eng.reset_sequence()
    eng.set_rng_position(0)
    eng.match(0, ups[1].data_ptr())
    nx, ny, cost, _ = engine_field(eng)
    NX, NY, H = oracle.match(F1, F2, sx, sy, N, 2, jf, double_prop, True, prm.search_dist(), normals)
    assert np.array_equal(nx, NX) and np.array_equal(ny, NY) and np.array_equal(cost, H)

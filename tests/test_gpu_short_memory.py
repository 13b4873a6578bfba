"""Where the device has room for an up-sampled image but not for its key image beside it,
contexts and batches are made all the same and give the same flows; with less they are
refused.  (Short memory is made by the allocator's test hook.)"""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
from briefmatch_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.fixture(autouse=True)
def _no_limit():
    yield
    bm.lib().bm_debug_alloc_limit(0)


def _image_bytes(prm, pattern):
    r = int(np.abs(np.asarray(pattern).astype(np.int64)).max())
    return (prm.sx + 2 * r) * (prm.sy + 2 * r) * 4


def _flow(eng, frames):
    eng.reset_sequence()
    eng.set_rng_position(0)
    eng.process_frame(frames[0])
    out = eng.process_frame(frames[1])
    up = eng.read_buffer(bm.BM_BUF_UP, np.float32, eng.params.sx * eng.params.sy)
    return [np.array(a) for a in (*out, up)]


@pytest.mark.parametrize("W,H,u,N", [(61, 37, 2.0, 31), (150, 92, 2.9, 32)])
def test_context(W, H, u, N):
    prm = bm.BMParams.derive(W, H, u, u, N=N)
    frames = synth.make_pair(6, W, H, 3.0)[:2]
    eng = bm.FlowEngine(prm)
    want = _flow(eng, frames)
    eng.clean()
    image = _image_bytes(prm, prm.make_pattern(0))
    bm.lib().bm_debug_alloc_limit(image)
    eng = bm.FlowEngine(prm)
    got = _flow(eng, frames)
    eng.clean()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    bm.lib().bm_debug_alloc_limit(image - 1)
    with pytest.raises(bm.CudaException, match="status %d: " % bm.BM_ERR_NOMEM):
        bm.FlowEngine(prm)


@pytest.mark.parametrize("N", [64, 200, 512])
def test_wider_pattern(N):
    W, H = 75, 46
    prm = bm.BMParams.derive(W, H, 2.0, 2.0, N=N)
    frames = synth.make_pair(7, W, H, 3.0)[:2]
    wide = np.clip(prm.make_pattern(5) * 40.0, -250, 250)
    eng = bm.FlowEngine(prm)
    eng.set_pattern(wide)
    want = _flow(eng, frames)
    eng.clean()
    eng = bm.FlowEngine(prm)
    bm.lib().bm_debug_alloc_limit(_image_bytes(prm, wide) - 1)
    with pytest.raises(bm.CudaException, match="status %d: " % bm.BM_ERR_NOMEM):
        eng.set_pattern(wide)
    bm.lib().bm_debug_alloc_limit(_image_bytes(prm, wide))
    eng.set_pattern(wide)
    got = _flow(eng, frames)
    eng.clean()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_batch():
    sizes = [(400, 301), (380, 290), (411, 222), (120, 88)]
    ups = [2.9, 2.5, 2.9, 1.0]
    params = [bm.BMParams.derive(w, h, u, u, N=32) for (w, h), u in zip(sizes, ups)]
    frames = [synth.make_pair(30 + k, w, h, 3.0)[:2] for k, (w, h) in enumerate(sizes)]
    images = sum(_image_bytes(p, p.make_pattern(0)) for p in params[:3])

    def flows(b):
        b.set_schedule(per_pair=1, use_graph=1, streams=2)
        b.load_frames(b.pack_frames(frames))
        b.run()
        b.synchronize()
        out = b.read_flows()
        b.close()
        return out

    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    b = bm.Batch(params)
    taken = before - torch.cuda.mem_get_info()[0]
    want = flows(b)
    # the smallest limit a batch can be made under
    lo, hi = 0, 2 * taken
    while hi - lo > 1:
        mid = (lo + hi) // 2
        bm.lib().bm_debug_alloc_limit(mid)
        try:
            bm.Batch(params).close()
            hi = mid
        except bm.CudaException as e:
            assert "status %d: " % bm.BM_ERR_NOMEM in str(e)
            lo = mid
    assert hi <= taken - images + (4 << 20)   # the device hands out memory 2 MB at a time
    bm.lib().bm_debug_alloc_limit(hi)
    b = bm.Batch(params)
    bm.lib().bm_debug_alloc_limit(0)
    for (gu, gv), (wu, wv) in zip(flows(b), want):
        assert np.array_equal(gu, wu) and np.array_equal(gv, wv)

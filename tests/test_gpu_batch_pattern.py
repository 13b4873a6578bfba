"""A pattern set after a batch's step was captured into its graph holds for the next run."""
from __future__ import annotations

import numpy as np
import pytest

import briefmatch_gb300 as bm
from briefmatch_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)


@pytest.mark.parametrize("kw", [dict(per_pair=1, streams=2), dict(per_pair=1, streams=1), dict(per_pair=0)])
@pytest.mark.parametrize("scale", [0.5, 3.0])   # inside the image's margin, and wider than it
def test_pattern_after_a_captured_run(kw, scale):
    sizes = [(61, 43), (52, 36)]
    params = [bm.BMParams.derive(w, h, 2.0, 1.5, N=64) for w, h in sizes]
    frames = [synth.make_pair(9 + k, w, h, 3.0)[:2] for k, (w, h) in enumerate(sizes)]
    b = bm.Batch(params)
    b.set_schedule(persistent=0, use_graph=1, **kw)
    b.load_frames(b.pack_frames(frames))
    b.run()
    b.synchronize()
    first = b.read_flows()
    pattern = params[1].make_pattern(12) * scale
    b.set_pattern(1, pattern)
    b.run()
    b.synchronize()
    got = b.read_flows()
    b.close()
    eng = bm.FlowEngine(params[1])
    eng.set_pattern(pattern)
    eng.process_frame(frames[1][0])
    want = eng.process_frame(frames[1][1])
    eng.clean()
    assert all(np.array_equal(x, y) for x, y in zip(got[0], first[0]))
    assert all(np.array_equal(x, y) for x, y in zip(got[1], want))
    assert not np.array_equal(got[1][0], first[1][0])

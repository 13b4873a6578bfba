"""Timing cases of the flow engine: the calls its users make, over the range of sizes
and options they are made with.

listed()  the named cases; draw(rng) one more case of the same ranges.
prepare(case, seed)  inputs on the GPU (or the host, for the host call) and the engine,
          batch or network a program keeps between calls.
run(state)  one pass through the public entry points and everything it returns.
work(case)  bytes and operations of one pass that the path cannot do without.
exact(case, seed)  the computed values in 64 bits, for the calls whose result is a
          formula of the inputs (refinement, up-sampling, network); the matched flow
          follows integer decisions and a random stream and has no such value.

The frames follow the synthetic generator's description (Gaussian blobs on mid-grey,
band-limited noise, affine flow plus rigid rectangles, sensor noise), evaluated on the
GPU so that preparing a case stays cheap.
"""
import math

import numpy as np
import torch

import briefmatch_gb300 as bm
from briefmatch_gb300 import learn, synth

# (iterations, jump maximum, input reduction) of the proposal-seeded schedules: the one
# calibrated on the 1024x436 sequences, and the batch's
SEQ_SEEDED = (1, 128, 1)
BATCH_SEEDED = (1, 32, 2)
TRAIN_W, TRAIN_H = 512, 384


def listed():
    return [
        # one small pair handed over as host arrays and read back, the call a camera
        # loop makes: launches, copies and latency
        {"name": "host_96x64_u1.5_N64", "kind": "host", "w": 96, "h": 64, "u": 1.5, "bits": 64},
        # a small pair at the command line's default up-sampling (2.74 x 3.052) and
        # feature length
        {"name": "pair_320x240_default_N128", "kind": "frames", "w": 320, "h": 240, "u": 0.0, "bits": 128, "frames": 2,
         "seeded": False, "pipelined": False},
        # the fast setting: short descriptors, little up-sampling
        {"name": "pair_584x388_u1.5_N32", "kind": "frames", "w": 584, "h": 388, "u": 1.5, "bits": 32, "frames": 2,
         "seeded": False, "pipelined": False},
        # a video: eight frames, pipelined, temporal initialisation -- the moderate setting
        {"name": "seq_1024x436_u2.9_N128", "kind": "frames", "w": 1024, "h": 436, "u": 2.9, "bits": 128, "frames": 8,
         "seeded": False, "pipelined": True},
        # the same video seeded by the learned proposal
        {"name": "seeded_1024x436_u2.9_N128", "kind": "frames", "w": 1024, "h": 436, "u": 2.9, "bits": 128, "frames": 8,
         "seeded": True, "pipelined": True},
        # the accurate setting: full-HD frames, 64-byte descriptors (the largest call)
        {"name": "pair_1920x1080_u4.9_N512", "kind": "frames", "w": 1920, "h": 1080, "u": 4.9, "bits": 512, "frames": 2,
         "seeded": False, "pipelined": False},
        # uneven pairs of a data set in one step, and the same seeded
        {"name": "batch_12_u2.9_N128", "kind": "batch", "pairs": 12, "sizes": 5, "u": 2.9, "bits": 128, "seeded": False},
        {"name": "batch_seeded_12_u2.9_N128", "kind": "batch", "pairs": 12, "sizes": 5, "u": 2.9, "bits": 128,
         "seeded": True},
        # refinement alone on a full-HD field the caller owns
        {"name": "refine_1920x1080", "kind": "refine", "w": 1920, "h": 1080, "sEPE": 0.4, "sI": 0.1, "median": 1.0,
         "spatial": 0.85},
        # the stage calls, on float images of an odd size with an odd feature length
        {"name": "stages_417x251_default_N100", "kind": "stages", "w": 417, "h": 251, "u": 0.0, "bits": 100,
         "both_ways": True, "philox": False},
        # the proposal network alone, and one of its training steps
        {"name": "proposal_1024x436", "kind": "proposal", "w": 1024, "h": 436, "reduce": 1},
        {"name": "train_512x384_B32", "kind": "train", "batch": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "frames", "frames", "frames", "batch", "refine", "stages", "proposal", "train"])
    if kind == "host":
        return {"kind": "host", "w": _log_int(rng, 64, 640), "h": _log_int(rng, 48, 480),
                "u": rng.choice([1.0, 1.5, 2.0, 2.9]), "bits": rng.choice([32, 64, 128])}
    if kind == "frames":
        seeded = rng.random() < 0.4
        w, h = _log_int(rng, 96, 1920), _log_int(rng, 64, 1080)
        u = rng.choice([1.0, 1.5, 0.0, 2.0, 2.9, 2.9, 4.9])
        return {"kind": "frames", "w": w, "h": h, "u": u, "bits": rng.choice([32, 64, 100, 128, 128, 256, 512]),
                "frames": min(rng.randint(2, 6), 1 + max(1, int(2e6 / (w * h)))), "seeded": seeded, "pipelined": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": "batch", "pairs": rng.randint(2, 12), "sizes": rng.randint(100, 10 ** 6),
                "u": rng.choice([1.5, 2.0, 2.9]), "bits": rng.choice([32, 64, 128, 128]), "seeded": rng.random() < 0.4}
    if kind == "refine":
        return {"kind": "refine", "w": _log_int(rng, 160, 1920), "h": _log_int(rng, 120, 1080),
                "sEPE": round(rng.uniform(0.2, 0.8), 3), "sI": round(rng.uniform(0.05, 0.2), 3),
                "median": rng.choice([0.5, 1.0, 1.0, 1.5]), "spatial": round(rng.uniform(0.4, 0.85), 3)}
    if kind == "stages":
        return {"kind": "stages", "w": _log_int(rng, 64, 640), "h": _log_int(rng, 48, 480),
                "u": rng.choice([0.0, 1.5, 2.0, 2.9]), "bits": rng.choice([31, 32, 64, 100, 128, 200]),
                "both_ways": rng.random() < 0.7, "philox": rng.random() < 0.3}
    if kind == "proposal":
        return {"kind": "proposal", "w": _log_int(rng, 128, 1920), "h": _log_int(rng, 96, 1080),
                "reduce": rng.choice([1, 1, 2])}
    return {"kind": "train", "batch": rng.randint(4, 32)}


# ---------------------------------------------------------------------------
# Synthetic frames on the GPU (elementwise operations only: the same seed gives the
# same bytes)
# ---------------------------------------------------------------------------
def _blur(img, sigma=3.0):
    r = int(math.ceil(3 * sigma))
    taps = [math.exp(-k * k / (2 * sigma * sigma)) for k in range(-r, r + 1)]
    total = sum(taps)
    for dim in (0, 1):
        n = img.shape[dim]
        idx = torch.arange(n, device=img.device)
        acc = torch.zeros_like(img)
        for k, t in zip(range(-r, r + 1), taps):
            acc += (t / total) * img.index_select(dim, (idx + k).clamp_(0, n - 1))
        img = acc
    return img


class _Scene:
    """Frames of one synthetic sequence: the first frame, then each frame warped from
    the one before by a newly drawn flow."""

    def __init__(self, seed, w, h, vmax):
        self.rng = np.random.default_rng(seed)
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
        self.w, self.h, self.vmax = w, h, vmax
        self.yy, self.xx = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
        img = torch.full((h, w), 128.0, device="cuda")
        for _ in range(40):
            cx, cy = self.rng.uniform(0, w), self.rng.uniform(0, h)
            s, a = self.rng.uniform(5, 40), self.rng.uniform(-80, 80)
            gx = torch.exp(-(self.xx[0] - cx) ** 2 / (2 * s * s))
            gy = torch.exp(-(self.yy[:, 0] - cy) ** 2 / (2 * s * s))
            img += (a * gy)[:, None] * gx[None, :]
        # noise of standard deviation 10 after a 3 px blur (which leaves
        # 1 / (2 sqrt(pi) 3) of white noise's)
        img += _blur(self._noise(10.0 * 2 * math.sqrt(math.pi) * 3.0))
        self.img = img

    def _noise(self, sigma):
        return torch.randn(self.h, self.w, device="cuda", generator=self.gen) * sigma

    def frame(self):
        return self.img.round().clamp(0, 255).to(torch.uint8)

    def flow(self):
        w, h, rng = self.w, self.h, self.rng
        t = rng.uniform(-1, 1, size=2)
        t *= rng.uniform(0, 4) / max(np.hypot(*t), 1e-9)
        ang, sc = math.radians(rng.uniform(-2, 2)), rng.uniform(0.97, 1.03)
        X, Y = self.xx - w / 2.0, self.yy - h / 2.0
        u = sc * (math.cos(ang) * X - math.sin(ang) * Y) - X + t[0]
        v = sc * (math.sin(ang) * X + math.cos(ang) * Y) - Y + t[1]
        for _ in range(int(rng.integers(3, 7))):
            rw, rh = rng.uniform(0.08, 0.3) * w, rng.uniform(0.08, 0.3) * h
            x0, y0 = int(rng.uniform(0, w - rw)), int(rng.uniform(0, h - rh))
            vel = rng.uniform(-1, 1, size=2)
            vel *= rng.uniform(0, self.vmax) / max(np.hypot(*vel), 1e-9)
            box = (slice(y0, y0 + int(rh) + 1), slice(x0, x0 + int(rw) + 1))
            u[box], v[box] = float(vel[0]), float(vel[1])
        return u, v

    def advance(self):
        """Moves to the next frame and returns the flow that led there."""
        u, v = self.flow()
        x, y = (self.xx - u).clamp_(0, self.w - 1), (self.yy - v).clamp_(0, self.h - 1)
        x0, y0 = x.floor(), y.floor()
        fx, fy = x - x0, y - y0
        x0, y0 = x0.long(), y0.long()
        x1, y1 = (x0 + 1).clamp_(max=self.w - 1), (y0 + 1).clamp_(max=self.h - 1)
        im = self.img
        nxt = ((1 - fx) * (1 - fy) * im[y0, x0] + fx * (1 - fy) * im[y0, x1] + (1 - fx) * fy * im[y1, x0]
               + fx * fy * im[y1, x1])
        self.img = (nxt + self._noise(2.0)).clamp_(0, 255)
        return u, v


def _frames(seed, w, h, n, vmax):
    s = _Scene(seed, w, h, vmax)
    out = [s.frame()]
    for _ in range(n - 1):
        s.advance()
        out.append(s.frame())
    return torch.stack(out)


def _vmax(case):
    return 24.0 if case["w"] > 1400 else 15.0 if case["w"] > 600 else 10.0


def _params(case, **kw):
    return bm.BMParams.derive(case["w"], case["h"], case["u"], case["u"], N=case["bits"], **kw)


class _State:
    """What a program keeps: its engine objects, inputs, outputs and a stream of its
    own that is ordered with torch's current stream around each pass."""

    def __init__(self, case, **kw):
        self.case = case
        self.stream = torch.cuda.Stream()
        self.__dict__.update(kw)

    def begin(self):
        self.stream.wait_stream(torch.cuda.current_stream())

    def end(self):
        torch.cuda.current_stream().wait_stream(self.stream)


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def _prepare_host(case, seed):
    frames = _frames(seed, case["w"], case["h"], 2, _vmax(case)).cpu().numpy()
    return _State(case, eng=bm.FlowEngine(_params(case)), frames=[np.ascontiguousarray(f) for f in frames])


def _attach_proposal(eng, case):
    it, jf, red = SEQ_SEEDED
    net = learn.load_net(learn.DEFAULT_WEIGHTS, 1, case["h"] // 4, case["w"] // 4)
    bm.set_proposal(eng, net, 0.5, it, jf)
    bm.set_proposal_reduce(eng, red)
    return net


def _prepare_frames(case, seed):
    w, h, n = case["w"], case["h"], case["frames"]
    frames = _frames(seed, w, h, n, _vmax(case))
    eng = bm.BriefMatch(_params(case))
    eng.setup()
    s = _State(case, eng=eng, frames=frames, flow=torch.empty(n - 1, 2, h, w, device="cuda"))
    eng.set_stream(s.stream.cuda_stream)
    s.net = _attach_proposal(eng, case) if case["seeded"] else None
    if case["pipelined"]:
        eng.set_pipelined(True)
    return s


def _batch_sizes(case):
    return synth.make_batch_sizes(case["sizes"], case["pairs"])


def _prepare_batch(case, seed):
    sizes = _batch_sizes(case)
    batch = bm.Batch([_params(dict(case, w=w, h=h)) for w, h in sizes])
    frames = torch.cat([_frames(seed * 1000 + k, w, h, 2, _vmax({"w": w})).reshape(-1) for k, (w, h) in enumerate(sizes)])
    s = _State(case, batch=batch, frames=frames, flows=torch.empty(batch.flows_bytes // 4, device="cuda"), net=None)
    batch.set_stream(s.stream.cuda_stream)
    if case["seeded"]:
        it, jf, red = BATCH_SEEDED
        s.net = learn.load_net(learn.DEFAULT_WEIGHTS, 1, max(h for _, h in sizes) // 4, max(w for w, _ in sizes) // 4)
        batch.set_proposal(s.net, 0.5, it, jf)
        batch.set_proposal_reduce(red)
    # the schedule the autotuner picks for such batches: pairs on two graph branches
    batch.set_schedule(per_pair=1, persistent=0, use_graph=1, streams=2)
    return s


def _refine_inputs(case, seed):
    """A field as matching leaves it (the true flow in steps of 1/3 px with noise and
    outliers) and its guide frame."""
    sc = _Scene(seed, case["w"], case["h"], _vmax(case))
    guide = sc.frame().float()
    planes = []
    for a in sc.flow():
        f = ((a + sc._noise(0.25)) * 3.0).round() / 3.0
        out = torch.rand(case["h"], case["w"], device="cuda", generator=sc.gen) < 0.02
        planes.append(torch.where(out, f + sc._noise(6.0), f).contiguous())
    return planes[0], planes[1], guide


def _refine_sizes(case):
    prm = bm.BMParams.derive(case["w"], case["h"], 2.9, 2.9, median_size=case["median"], range_spatial=case["spatial"])
    return int(prm.fsize), float(prm.sS)


def _prepare_refine(case, seed):
    u, v, guide = _refine_inputs(case, seed)
    fsize, sS = _refine_sizes(case)
    return _State(case, u=u, v=v, guide=guide, out=torch.empty(2, case["h"], case["w"], device="cuda"), fsize=fsize, sS=sS)


def _stage_frames(case, seed):
    return _frames(seed, case["w"], case["h"], 2, _vmax(case)).float()


def _prepare_stages(case, seed):
    prm = _params(case, doubleProp=int(case["both_ways"]),
                  rng=bm.BM_RNG_PHILOX if case["philox"] else bm.BM_RNG_XORWOW, seed=9)
    eng = bm.BriefMatch(prm)
    eng.setup()
    n = (prm.sy, prm.sx)
    s = _State(case, eng=eng, frames=_stage_frames(case, seed), up=torch.empty(2, *n, device="cuda"),
               nx=torch.empty(n, dtype=torch.int16, device="cuda"), ny=torch.empty(n, dtype=torch.int16, device="cuda"),
               dist=torch.empty(n, device="cuda"))
    eng.set_stream(s.stream.cuda_stream)
    return s


def _cells(case):
    return case["h"] // case["reduce"] // 4, case["w"] // case["reduce"] // 4


def _prepare_proposal(case, seed):
    h4, w4 = _cells(case)
    return _State(case, frames=_frames(seed, case["w"], case["h"], 2, _vmax(case)),
                  net=learn.load_net(learn.DEFAULT_WEIGHTS, 1, h4, w4), out=torch.empty(1, h4, w4, 3, device="cuda"))


def _train_inputs(case, seed):
    B = case["batch"]
    f0 = torch.empty(B, TRAIN_H, TRAIN_W, dtype=torch.uint8, device="cuda")
    f1 = torch.empty_like(f0)
    target = torch.empty(B, TRAIN_H // 4, TRAIN_W // 4, 3, device="cuda")
    sc = None
    for b in range(B):
        if b % 8 == 0:
            sc = _Scene(seed * 1000 + b, TRAIN_W, TRAIN_H, 15.0)
        f0[b] = sc.frame()
        uv = torch.stack(sc.advance(), -1)
        f1[b] = sc.frame()
        cell = uv.reshape(TRAIN_H // 4, 4, TRAIN_W // 4, 4, 2).mean((1, 3)) / 4.0
        target[b, ..., :2] = cell
        # the weight a forward-backward check leaves a cell: most count in full
        target[b, ..., 2] = (torch.rand(cell.shape[:2], device="cuda", generator=sc.gen) * 1.5).clamp_(max=1.0)
    return f0, f1, target


def _prepare_train(case, seed):
    f0, f1, target = _train_inputs(case, seed)
    net = learn.load_net(learn.DEFAULT_WEIGHTS, case["batch"], TRAIN_H // 4, TRAIN_W // 4)
    s = _State(case, f0=f0, f1=f1, target=target, net=net, grad=torch.empty(net.nparam, device="cuda"))
    net.snapshot(0, s.stream.cuda_stream)
    return s


def prepare(case, seed):
    s = {"host": _prepare_host, "frames": _prepare_frames, "batch": _prepare_batch, "refine": _prepare_refine,
         "stages": _prepare_stages, "proposal": _prepare_proposal, "train": _prepare_train}[case["kind"]](case, seed)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def _run_host(s):
    s.eng.reset_sequence()
    s.eng.set_rng_position(0)
    s.eng.process_frame(s.frames[0])
    return s.eng.process_frame(s.frames[1])


def _run_frames(s):
    eng = s.eng
    s.begin()
    eng.reset_sequence()
    eng.set_rng_position(0)
    eng.frame(s.frames[0].data_ptr(), True)
    for k in range(1, s.frames.shape[0]):
        eng.frame(s.frames[k].data_ptr(), True, s.flow[k - 1, 0].data_ptr(), s.flow[k - 1, 1].data_ptr(), True)
    eng.join()
    s.end()
    return s.flow


def _run_batch(s):
    s.begin()
    s.batch.load_frames(s.frames.data_ptr(), on_device=True)
    s.batch.run()
    s.batch.read_flows_into(s.flows.data_ptr(), True)
    s.end()
    return s.flows


def _run_refine(s):
    c = s.case
    s.begin()
    bm.refine_noalloc(s.u.data_ptr(), s.v.data_ptr(), s.guide.data_ptr(), s.out[0].data_ptr(), s.out[1].data_ptr(),
                      c["w"], c["h"], s.fsize, c["sEPE"], c["sI"], s.sS, s.stream.cuda_stream)
    s.end()
    return s.out


def _run_stages(s):
    eng = s.eng
    s.begin()
    eng.reset_sequence()
    eng.set_rng_position(0)
    eng.upsample(s.frames[0].data_ptr(), s.up[0].data_ptr())
    eng.features(s.up[0].data_ptr(), 0)
    eng.upsample(s.frames[1].data_ptr(), s.up[1].data_ptr())
    eng.match(s.up[0].data_ptr(), s.up[1].data_ptr())
    eng.downsample()
    eng.process(s.frames[0].data_ptr())
    eng.export_field(s.nx.data_ptr(), s.ny.data_ptr(), s.dist.data_ptr())
    u, v = eng.convert()
    s.end()
    return [s.up[1], s.nx, s.ny, s.dist, u, v]


def _run_proposal(s):
    c = s.case
    h4, w4 = _cells(c)
    s.begin()
    s.net.prepare(0, s.frames[0].data_ptr(), s.frames[1].data_ptr(), c["w"], c["h"], s.stream.cuda_stream, c["reduce"])
    s.net.forward(1, h4, w4, s.out.data_ptr(), s.stream.cuda_stream)
    s.end()
    return s.out


def _run_train(s):
    B, st = s.case["batch"], s.stream.cuda_stream
    s.begin()
    # every pass steps from the same weights, so that its gradient is the same
    s.net.restore(0, st)
    for b in range(B):
        s.net.prepare(b, s.f0[b].data_ptr(), s.f1[b].data_ptr(), TRAIN_W, TRAIN_H, st)
    loss = s.net.train_step(B, TRAIN_H // 4, TRAIN_W // 4, s.target.data_ptr(), 2e-3, s.grad.data_ptr(), st)
    s.end()
    return [s.grad, loss]


def run(state):
    return {"host": _run_host, "frames": _run_frames, "batch": _run_batch, "refine": _run_refine, "stages": _run_stages,
            "proposal": _run_proposal, "train": _run_train}[state.case["kind"]](state)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _tri_ops(w, h, sS):
    s = math.ceil(2.5 * sS)
    return 16.0 * w * h * (2 * s) ** 2


def _pair_ops(prm, new_frames, seeded):
    """Operations of one matched pair: per up-sampled pixel of each new frame the 36
    multiply-adds of the up-sampling and one comparison per descriptor bit; per pixel
    and candidate a word-wise XOR, popcount and add; the trilateral filter."""
    n, ns = float(prm.sx) * prm.sy, (prm.N + 31) // 32
    it, jf = (SEQ_SEEDED[0], SEQ_SEEDED[1]) if seeded else (prm.iterations, prm.jfMax)
    candidates = 1 + it * (4 * (int(math.log2(jf)) + 1) + 1)
    ups = 72.0 if prm.sx != prm.sx_in else 0.0
    return new_frames * n * (ups + prm.N) + n * candidates * 3 * ns + _tri_ops(prm.sx_in, prm.sy_in, prm.sS)


def _net_flops(cells):
    return 2.0 * 9 * (5 * 32 * 32 + 32 * 3) * cells


def work(case):
    kind = case["kind"]
    if kind in ("host", "frames", "stages"):
        prm = _params(case)
        pairs = case.get("frames", 2) - 1
        ni, seeded = float(case["w"]) * case["h"], case.get("seeded", False)
        ops = pairs * _pair_ops(prm, (pairs + 1.0) / pairs, seeded)
        if seeded:
            ops += pairs * _net_flops(ni / 16)
        bytes_ = (pairs + 1) * ni * (4 if kind == "stages" else 1) + pairs * ni * 8
        if kind == "stages":
            bytes_ += float(prm.sx) * prm.sy * (2 * 4 + 2 + 2 + 4)
        return {"bytes": bytes_, "flops": ops}
    if kind == "batch":
        ops = bytes_ = 0.0
        for w, h in _batch_sizes(case):
            ops += _pair_ops(_params(dict(case, w=w, h=h)), 2, case["seeded"])
            ops += _net_flops(w * h / 64.0) if case["seeded"] else 0.0
            bytes_ += w * h * (2 + 8.0)
        return {"bytes": bytes_, "flops": ops}
    if kind == "refine":
        return {"bytes": case["w"] * case["h"] * 20.0, "flops": _tri_ops(case["w"], case["h"], _refine_sizes(case)[1])}
    if kind == "proposal":
        h4, w4 = _cells(case)
        return {"bytes": 2.0 * case["w"] * case["h"] + 12.0 * h4 * w4, "flops": _net_flops(h4 * w4)}
    cells = case["batch"] * (TRAIN_W // 4) * (TRAIN_H // 4)
    # both frames and the targets in, the gradient out; forward and weight gradient of
    # every layer, data gradient of all but the first
    return {"bytes": cells * 44.0 + 4.0 * 47107, "flops": 3 * _net_flops(cells) - 2.0 * 9 * 32 * 32 * cells}


# ---------------------------------------------------------------------------
# exact: 64-bit values by plain torch
# ---------------------------------------------------------------------------
def _exact_median(p, fsize):
    """Median over linear indices along rows, then down columns, zeros outside."""
    h, w = p.shape
    ks = fsize // 2
    flat = torch.cat([p.new_zeros(ks), p.reshape(-1), p.new_zeros(fsize)])
    rows = flat.unfold(0, fsize, 1)[:h * w]
    p = torch.cat([c.sort(dim=1).values[:, ks] for c in rows.split(1 << 18)]).reshape(h, w)
    tall = torch.cat([p.new_zeros(ks, w), p, p.new_zeros(fsize, w)])
    cols = tall.unfold(0, fsize, 1)[:h]
    return torch.cat([c.sort(dim=2).values[..., ks] for c in cols.split(128)])


def _exact_refine(case, seed):
    u, v, guide = (p.double() for p in _refine_inputs(case, seed))
    fsize, sS = _refine_sizes(case)
    um, vm = _exact_median(u, fsize), _exact_median(v, fsize)
    s = math.ceil(2.5 * sS)
    sq = lambda x: float(np.float32(x) * np.float32(x))  # noqa: E731
    cE, cI, cS = 1 / (2 * sq(case["sEPE"])), 1 / (2 * sq(case["sI"]) * 255.0 ** 2), 1 / (2 * sq(sS))
    h, w = u.shape

    def padded(p):
        iy = torch.arange(-s, h + s, device="cuda").clamp_(0, h - 1)
        ix = torch.arange(-s, w + s, device="cuda").clamp_(0, w - 1)
        return p[iy][:, ix].contiguous()

    U, V, G = padded(u), padded(v), padded(guide)
    uf, vf, W = torch.zeros_like(u), torch.zeros_like(u), torch.zeros_like(u)
    for j in range(2 * s):
        for i in range(2 * s):
            u1, v1 = U[j:j + h, i:i + w], V[j:j + h, i:i + w]
            e = (u1 - um).square_().add_((v1 - vm).square_()).mul_(-cE)
            e.add_((G[j:j + h, i:i + w] - guide).square_(), alpha=-cI).sub_(cS * ((i - s) ** 2 + (j - s) ** 2))
            e.exp_()
            uf.addcmul_(e, u1)
            vf.addcmul_(e, v1)
            W.add_(e)
    W.clamp_(min=1e-5)
    return torch.stack([uf / W, vf / W])


def _exact_upsample(img, sx, sy):
    def weights(n_in, n_out):
        xp = torch.arange(n_out, device="cuda", dtype=torch.float64) * n_in / n_out
        first = xp.floor().long()
        k = first[:, None] + torch.arange(-2, 4, device="cuda")
        x = math.pi * (xp[:, None] - k)
        lw = torch.where(x == 0, torch.ones_like(x), 3 * torch.sin(x) * torch.sin(x / 3) / (x * x))
        return lw, k.clamp(0, n_in - 1)

    h, w = img.shape
    lx, ix = weights(w, sx)
    ly, iy = weights(h, sy)
    rows = (img.double()[iy] * ly[:, :, None]).sum(1) / ly.sum(1)[:, None]
    return (rows[:, ix] * lx[None]).sum(2) / lx.sum(1)[None]


def _net_params():
    """The committed weights as double tensors [(W cout x cin x 3 x 3, b)]."""
    flat = torch.from_numpy(np.fromfile(learn.DEFAULT_WEIGHTS, np.float32)).double().cuda()
    return flat


def _net_forward(flat, f0, f1):
    """[B][h4][w4][3] of the network on frames f0, f1 ([B][h][w], double, 0..255)."""
    x = torch.cat([torch.nn.functional.pixel_unshuffle(f[:, None] / 127.5 - 1.0, 4) for f in (f0, f1)], 1)
    at = 0
    for cout, dil in ((32, 1), (32, 2), (32, 4), (32, 8), (32, 1), (3, 1)):
        n = cout * 9 * 32
        wgt = flat[at:at + n].reshape(cout, 3, 3, 32).permute(0, 3, 1, 2)
        x = torch.nn.functional.conv2d(x, wgt, flat[at + n:at + n + cout], padding=dil, dilation=dil)
        at += n + cout
        if cout == 32:
            x = x.relu()
    return x.permute(0, 2, 3, 1)


def _exact_proposal(case, seed):
    red = case["reduce"]
    f = _frames(seed, case["w"], case["h"], 2, _vmax(case)).double()
    h4, w4 = _cells(case)
    f = f[:, :h4 * 4 * red, :w4 * 4 * red]
    if red > 1:  # each reduced pixel is a rounded byte
        f = f.reshape(2, h4 * 4, red, w4 * 4, red).mean((2, 4)).round()
    with torch.no_grad():
        return _net_forward(_net_params(), f[:1], f[1:])


def _exact_train(case, seed):
    f0, f1, target = _train_inputs(case, seed)
    flat = _net_params().requires_grad_()
    t = target.double()
    cells = t[..., 0].numel()
    F = torch.nn.functional
    for b in range(0, case["batch"], 4):
        out = _net_forward(flat, f0[b:b + 4].double(), f1[b:b + 4].double())
        tb = t[b:b + 4]
        near = (out[..., :2] - tb[..., :2]).abs().sum(-1).detach() < 1.0
        lf = F.smooth_l1_loss(out[..., :2], tb[..., :2], reduction="none").sum(-1)
        lc = F.binary_cross_entropy_with_logits(out[..., 2], near.double(), reduction="none")
        (((lf + 0.25 * lc) * tb[..., 2]).sum() / cells).backward()
    return [flat.grad, None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "refine":
        return _exact_refine(case, seed)
    if kind == "stages":
        prm = _params(case)
        return [_exact_upsample(_stage_frames(case, seed)[1], prm.sx, prm.sy), None, None, None, None, None]
    if kind == "proposal":
        return _exact_proposal(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    return None

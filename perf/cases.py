"""The work a user of floodca_b200 has it do, as measurable cases.

Five kinds of case, each through a public entry point:

  ca     a scenario on a resident session: upload the start depth, reset the
         clock, run the given number of steps, download h, hmax and tmax
         (floodca_b200.sim.Session and the fcab_sim_* calls it wraps). One
         session serves many scenarios, as the reference's ensemble session
         does.
  dropin the reference-facing fca_cuda_run on host buffers: one whole call
         (set-up, uploads, steps, downloads) through sim.DropinGrid.
  batch  an ensemble of grids of different sizes advanced together
         (floodca_b200.ensemble.Batch), every member's depths downloaded.
  unet   the surrogate on images: a forward pass (MC dropout, as the
         screening of an ensemble runs it, or deterministic), or a forward
         and backward pass that leaves every weight gradient.
  conv   one 3x3 convolution layer of the surrogate: forward with bias and
         ReLU, data gradient, weight gradient.

Grids are the recipe of floodca_b200.synth (a plane falling to the south,
fractal relief, a carved channel, six Manning classes in patches), made on
the GPU from the seed. `exact` restates the step and the layers in 64-bit
torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from floodca_b200 import ensemble, synth
from floodca_b200.lib import check, core
from floodca_b200.sim import Domain, DropinGrid, RunParams, Session
from floodca_b200.unet import UNet

DX = 90.0
F64 = torch.float64

# (input channels, output channels) of the surrogate's layers with a data gradient
CONV_PAIRS = ((32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 256), (256, 256),
              (384, 128), (192, 64), (96, 32))


def listed():
    ca = {"kind": "ca", "K": 4, "prec": "f32", "mask": "land", "rain": "box", "edges": "south",
          "warm": True, "inflow": False}
    return [
        # a small catchment with sea and wall cells: launch and step latency are all there is
        dict(ca, name="ca small coast 61x93", rows=61, cols=93, steps=300, mask="coast",
             rain="field", edges="all", warm=False),
        # the 256 x 256 town grid of the benchmark set, dry start, a whole 2 h run's steps
        dict(ca, name="ca 256 storm", rows=256, cols=256, steps=295, warm=False),
        # a coastal district as the reference's own rasters have it: SEA and
        # WALL cells, a rain field under the triangular hyetograph, all edges open
        dict(ca, name="ca coast 733x1101", rows=733, cols=1101, steps=300, mask="coast",
             rain="field", edges="all", warm=False),
        # the 2048 x 2048 rainstorm of the benchmark set
        dict(ca, name="ca 2048 storm", rows=2048, cols=2048, steps=300),
        # the benchmark grid itself: 4096 x 4096 with a point inflow
        dict(ca, name="ca 4096 inflow", rows=4096, cols=4096, steps=300, inflow=True),
        # eight neighbours, ragged sides
        dict(ca, name="ca K8 1003x1498", rows=1003, cols=1498, steps=200, K=8),
        # the FP64 build's precision
        dict(ca, name="ca f64 511x770", rows=511, cols=770, steps=100, prec="f64"),
        # one call of the reference's CUDA entry point on host buffers
        {"kind": "dropin", "name": "dropin 1024x1024", "rows": 1024, "cols": 1024, "steps": 400},
        # an ensemble of 24 catchments of 256..1024 cells a side
        {"kind": "batch", "name": "batch of 24", "members": 24, "lo": 256, "hi": 1024,
         "steps": 100},
        # one screening pass of the surrogate: 64 images, dropout on
        {"kind": "unet", "name": "unet screening 64x256x256", "images": 64, "rows": 256,
         "cols": 256, "mc": True, "grad": False},
        # a training batch of the surrogate up to its gradients
        {"kind": "unet", "name": "unet gradients 32x256x256", "images": 32, "rows": 256,
         "cols": 256, "mc": True, "grad": True},
        # one layer of the surrogate by itself, ragged images
        {"kind": "conv", "name": "conv 64 to 128 17x61x67", "images": 17, "rows": 61, "cols": 67,
         "cin": 64, "cout": 128},
    ]


def _log(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("ca", "ca", "ca", "ca", "dropin", "batch", "unet", "unet", "conv"))
    if kind == "ca":
        prec = "f64" if rng.random() < 0.15 else "f32"
        mask = rng.choice(("land", "land", "coast"))
        top = 1024 if prec == "f64" else 4096
        rows, cols = _log(rng, 48, top), _log(rng, 48, top)
        K = rng.choice((4, 4, 8))
        most = min(300, int((2e7 if prec == "f64" else 1.2e9) / (rows * cols)))
        steps = _log(rng, min(40, most), max(41, most)) if most >= 1 else 1
        return {"kind": "ca", "rows": rows, "cols": cols, "steps": steps, "K": K, "prec": prec,
                "mask": mask, "rain": "field" if mask == "coast" else "box",
                "edges": rng.choice(("south", "all", "none")), "warm": rng.random() < 0.5,
                "inflow": rng.random() < 0.3}
    if kind == "dropin":
        return {"kind": "dropin", "rows": _log(rng, 64, 1500), "cols": _log(rng, 64, 1500),
                "steps": _log(rng, 100, 400)}
    if kind == "batch":
        lo = _log(rng, 128, 512)
        return {"kind": "batch", "members": rng.randint(4, 24), "lo": lo,
                "hi": min(1024, lo * rng.randint(1, 4)), "steps": _log(rng, 30, 100)}
    if kind == "unet":
        return {"kind": "unet", "images": rng.choice((1, 2, 5, 8, 16, 24, 32)),
                "rows": 8 * rng.randint(8, 32), "cols": 8 * rng.randint(8, 32),
                "mc": rng.random() < 0.5, "grad": rng.random() < 0.5}
    cin, cout = rng.choice(CONV_PAIRS)
    return {"kind": "conv", "images": rng.randint(1, 32), "rows": _log(rng, 8, 128),
            "cols": _log(rng, 8, 128), "cin": cin, "cout": cout}


# --------------------------------------------------------------------------
# Inputs.

def _terrain(rows, cols, gen):
    """Elevation and Manning n, float64 on the GPU."""
    ky = torch.fft.fftfreq(rows, device="cuda", dtype=F64)[:, None]
    kx = torch.fft.rfftfreq(cols, device="cuda", dtype=F64)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amp = k ** -1.7
    amp[0, 0] = 0.0
    phase = torch.rand(amp.shape, generator=gen, device="cuda", dtype=F64) * (2 * math.pi)
    f = torch.fft.irfft2(torch.polar(amp, phase), s=(rows, cols))
    f = f - f.mean()
    f = f * (10.0 / f.abs().max())
    r = torch.arange(rows, device="cuda", dtype=F64)[:, None]
    z = 10.0 + 0.005 * DX * (rows - 1 - r) + f
    c0 = cols // 2 - 1
    z[:, c0:c0 + 3] -= 2.0
    nclass = len(synth.MANNING_CLASSES)
    cls = torch.randint(0, nclass, (rows // 48 + 1, cols // 48 + 1), generator=gen, device="cuda")
    cls = cls.repeat_interleave(48, 0).repeat_interleave(48, 1)[:rows, :cols]
    return z, torch.tensor(synth.MANNING_CLASSES, device="cuda", dtype=F64)[cls]


def _scenario(case, seed):
    """The fields (GPU tensors of the precision's type) and run parameters of
    a ca case."""
    rows, cols = case["rows"], case["cols"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dt = F64 if case["prec"] == "f64" else torch.float32
    z, n = _terrain(rows, cols, gen)
    n = n * float(torch.empty(1).uniform_(0.7, 1.4, generator=torch.Generator().manual_seed(seed)))
    mask = torch.zeros((rows, cols), dtype=torch.uint8, device="cuda")
    if case["mask"] == "coast":
        # sea along a wavy south-west shore, walls in scattered blocks
        rr = torch.arange(rows, device="cuda", dtype=F64)[:, None] / rows
        cc = torch.arange(cols, device="cuda", dtype=F64)[None, :] / cols
        shore = 0.9 + 0.06 * torch.sin(9.0 * cc + seed % 7)
        mask[(rr > shore) | (cc < 0.06 * torch.sin(7.0 * rr) + 0.02)] = 1
        block = torch.rand((rows // 6 + 1, cols // 6 + 1), generator=gen, device="cuda") < 0.02
        block = block.repeat_interleave(6, 0).repeat_interleave(6, 1)[:rows, :cols]
        mask[block & (mask == 0)] = 2
    p = RunParams(K=case["K"], T_sim=10 * 86400.0, steps=case["steps"], out_every=600.0)
    if case["edges"] == "none":
        p = p.with_(boundary="closed")
    elif case["edges"] == "south":
        p = p.with_(edges=(0, 1, 0, 0))
    one = torch.ones((rows, cols), device="cuda", dtype=dt)
    if case["rain"] == "box":
        mm_h = float(torch.empty(1).uniform_(30.0, 100.0, generator=torch.Generator().manual_seed(
            seed + 1)))
        p = p.with_(hyeto="uniform", rain_end=7200.0)
        rday = one * (mm_h * 24.0 / 1000.0)
        runoff = one
    else:
        p = p.with_(hyeto="triangle", D_h=6.0, phi=0.4)
        w = torch.rand((rows // 64 + 2, cols // 64 + 2), generator=gen, device="cuda", dtype=F64)
        w = torch.nn.functional.interpolate(w[None, None], size=(rows, cols), mode="bilinear",
                                            align_corners=True)[0, 0]
        rday = (0.35 * w).to(dt)
        runoff = torch.where(n > 0.08, 0.55, 0.8).to(dt)
    if case["inflow"]:
        at = cols // 2
        p = p.with_(inflow_cell=at, inflow_peak=500.0, inflow_t_peak=10800.0,
                    inflow_t_end=21600.0)
        mask[0, at] = 0
    h = torch.full((rows, cols), 0.02 if case["warm"] else 0.0, device="cuda", dtype=dt)
    h = h * (0.5 + torch.rand((rows, cols), generator=gen, device="cuda", dtype=F64)).to(dt)
    return {"z": z.to(dt), "n": n.to(dt), "C": runoff, "R": rday.contiguous(), "mask": mask,
            "h": h.contiguous(), "p": p}


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _dev(t):
    return C.c_void_p(t.data_ptr())


class _Resident:
    """A session, its start depth and the host arrays its results go to."""

    def __init__(self, shape, p, z, h, mask, n, Cf, R, prec="f32"):
        torch.cuda.synchronize()
        self.s = Session.from_device(shape, DX, p, z, h, mask, n=n, Cf=Cf, Rday=R, precision=prec)
        self.h0 = h.cpu().numpy()
        self.out = [np.zeros_like(self.h0) for _ in range(3)]

    def restart(self):
        L, s = self.s.L, self.s
        check(L.fcab_sim_upload_state(s.h, _ptr(self.h0), None, None), "upload_state")
        check(L.fcab_sim_reset_time(s.h, 0.0, 0, 0.0, -1), "reset_time")

    def download(self):
        h, hmax, tmax = self.out
        check(self.s.L.fcab_sim_download(self.s.h, _ptr(h), _ptr(hmax), _ptr(tmax)), "download")


def _dropin_fields(case, seed):
    return _scenario({"rows": case["rows"], "cols": case["cols"], "steps": case["steps"], "K": 4,
                      "prec": "f32", "mask": "land", "rain": "field", "edges": "all",
                      "warm": False, "inflow": False}, seed)


def _batch_cases(case, seed):
    """The members of a batch, as ca cases."""
    top = max(case["hi"], case["lo"] + 1)
    return [({"rows": int(a), "cols": int(b), "steps": case["steps"], "K": 4, "prec": "f32",
              "mask": "land", "rain": "box", "edges": "south", "warm": False, "inflow": False},
             seed * 101 + i)
            for i, (a, b) in enumerate(_sides(case, top))]


def _sides(case, top):
    """Sides of a batch's members, the same for every seed (they decide the work)."""
    rng = np.random.default_rng(case["members"] * 1000 + case["lo"])
    return rng.integers(case["lo"], top, size=(case["members"], 2))


def _images(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    shape = (case["images"], case["rows"], case["cols"])
    x = torch.empty(shape + (4,), device="cuda")
    x[..., 0] = torch.randn(shape, generator=gen, device="cuda")
    x[..., 1] = 0.2 + 1.3 * torch.rand(shape, generator=gen, device="cuda")
    x[..., 2:] = torch.rand((shape[0], 1, 1, 2), generator=gen, device="cuda")
    t = torch.rand(shape, generator=gen, device="cuda") * 2.0
    return x, t


def _conv_inputs(case, seed):
    """Float32 images and weights with bf16 values, and a float32 bias."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    N, H, W, ci, co = (case[k] for k in ("images", "rows", "cols", "cin", "cout"))
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    bf = lambda t: t.to(torch.bfloat16).float()  # noqa: E731
    return (bf(rnd(N, H, W, ci)), bf(rnd(N, H, W, co)), bf(rnd(co, 9, ci) / math.sqrt(9 * ci)),
            rnd(co))


def _bordered(x):
    N, H, W, c = x.shape
    m = torch.zeros((N, H + 2, W + 2, c), dtype=torch.bfloat16, device="cuda")
    m[:, 1:-1, 1:-1] = x
    return m.view(-1, c)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ca":
        f = _scenario(case, seed)
        shape = (case["rows"], case["cols"])
        return {"case": case, "run": _Resident(shape, f["p"], f["z"], f["h"], f["mask"], f["n"],
                                               f["C"], f["R"], case["prec"])}
    if kind == "dropin":
        f = _dropin_fields(case, seed)
        host = {k: f[k].cpu().numpy() for k in ("z", "n", "C", "R", "mask", "h")}
        g = DropinGrid(Domain(z=host["z"], mask=host["mask"], n=host["n"], C=host["C"],
                              Rday=host["R"], h=host["h"], dx=DX), f["p"])
        return {"case": case, "g": g, "h0": host["h"], "acc0": bytes(g.acc)}
    if kind == "batch":
        members = []
        for c, s in _batch_cases(case, seed):
            f = _scenario(c, s)
            members.append(_Resident((c["rows"], c["cols"]), f["p"], f["z"], f["h"], f["mask"],
                                     f["n"], f["C"], f["R"]))
        b = ensemble.Batch([m.s for m in members], 2, 0,
                           [ensemble.seg_for(max(m.h0.shape), ensemble.DEFAULT_TUNING)
                            for m in members])
        return {"case": case, "members": members, "batch": b}
    if kind == "unet":
        x, t = _images(case, seed)
        model = UNet(seed=seed % 1000)
        model.prep()
        return {"case": case, "model": model, "x": x, "t": t, "drop": seed % 1000 + 1}
    x, dy, w, b = _conv_inputs(case, seed)
    N, H, W, ci, co = (case[k] for k in ("images", "rows", "cols", "cin", "cout"))
    rows = N * (H + 2) * (W + 2)
    st = {"case": case, "x": _bordered(x), "dy": _bordered(dy), "b": b,
          "wb": torch.empty((co, 9, ci), dtype=torch.bfloat16, device="cuda"),
          "wt": torch.empty((ci, 9, co), dtype=torch.bfloat16, device="cuda"),
          "y": torch.zeros((rows, co), dtype=torch.bfloat16, device="cuda"),
          "dx": torch.zeros((rows, ci), dtype=torch.bfloat16, device="cuda"),
          "dw": torch.zeros((co, 9, ci), device="cuda")}
    w = w.contiguous()
    check(core().fcab_unet_prep_weights(_dev(w), _dev(st["wb"]), _dev(st["wt"]), co, ci, None),
          "prep_weights")
    torch.cuda.synchronize()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ca":
        r = state["run"]
        r.restart()
        r.s.run()
        r.download()
        return {"h": r.out[0], "hmax": r.out[1], "tmax": r.out[2]}
    if kind == "dropin":
        g = state["g"]
        np.copyto(g.arrays["h"], state["h0"])
        np.copyto(g.arrays["hmax"], state["h0"])
        g.arrays["tmax"].fill(0.0)
        C.memmove(C.byref(g.acc), state["acc0"], len(state["acc0"]))
        if g.run() != 0:
            raise RuntimeError("fca_cuda_run failed")
        return {"h": g.arrays["h"], "hmax": g.arrays["hmax"], "tmax": g.arrays["tmax"],
                "steps": int(g.acc.step)}
    if kind == "batch":
        for m in state["members"]:
            m.restart()
        state["batch"].run(window=0.0)
        for m in state["members"]:
            m.download()
        return {"h": [m.out[0] for m in state["members"]],
                "hmax": [m.out[1] for m in state["members"]]}
    if kind == "unet":
        model = state["model"]
        out = model.forward(state["x"], dropout_seed=state["drop"] if case["mc"] else None)
        if not case["grad"]:
            return {"out": out}
        model.backward(state["t"])
        return {"out": out, "loss": model.loss_sum, "dhw": model.dhw, "dhb": model.dhb,
                "dw": [c.dw for c in model.convs()], "db": [c.db for c in model.convs()]}
    L = core()
    N, H, W, ci, co = (case[k] for k in ("images", "rows", "cols", "cin", "cout"))
    s = state
    check(L.fcab_unet_conv_fwd(_dev(s["x"]), N, H, W, ci, _dev(s["wb"]), co, _dev(s["b"]), 1,
                               _dev(s["y"]), None), "conv_fwd")
    check(L.fcab_unet_conv_dgrad(_dev(s["dy"]), N, H, W, co, _dev(s["wt"]), ci, _dev(s["dx"]),
                                 None), "conv_dgrad")
    s["dw"].zero_()        # the weight gradient adds into its output
    check(L.fcab_unet_conv_wgrad(_dev(s["dy"]), _dev(s["x"]), N, H, W, ci, co, _dev(s["dw"]),
                                 None), "conv_wgrad")
    return {"y": s["y"], "dx": s["dx"], "dw": s["dw"]}


# --------------------------------------------------------------------------
# What a pass cannot do without.

def _ca_work(cells, steps, K, size):
    """Each step of a run reads z, h, n and hmax and writes h and hmax (24
    bytes a cell in FP32); a face takes about 30 operations, a cell's
    limiter, update and stable velocity 40. The initial depth goes up and h,
    hmax, tmax come down once."""
    return {"bytes": cells * (steps * 6 + 4) * size, "flops": cells * steps * (30.0 * K / 2 + 40)}


def _unet_convs(case):
    """(pixels, input channels, output channels) of the surrogate's convolutions."""
    ch = (32, 64, 128, 256)
    px = [case["images"] * (case["rows"] >> k) * (case["cols"] >> k) for k in range(4)]
    out = [(px[0], 4, 32), (px[0], 32, 32)]
    for k in (1, 2, 3):
        out += [(px[k], ch[k - 1], ch[k]), (px[k], ch[k], ch[k])]
    for k in (2, 1, 0):
        out += [(px[k], ch[k + 1] + ch[k], ch[k]), (px[k], ch[k], ch[k])]
    return out


def work(case):
    kind = case["kind"]
    if kind in ("ca", "dropin"):
        return _ca_work(case["rows"] * case["cols"], case["steps"], case.get("K", 4),
                        8 if case.get("prec") == "f64" else 4)
    if kind == "batch":
        cells = sum(int(a) * int(b) for a, b in _sides(case, max(case["hi"], case["lo"] + 1)))
        return _ca_work(cells, case["steps"], 4, 4)
    if kind == "unet":
        convs = _unet_convs(case)
        px = convs[0][0]
        passes = 3 if case["grad"] else 1
        weights = sum(9 * a * b for _, a, b in convs) + 33
        # inputs, weights, the prediction; for gradients also every layer's
        # kept output (written once, read once), the target and the gradients
        kept = sum(p * b * 2 for p, _, b in convs) * 2 if case["grad"] else 0
        return {"bytes": px * (16 + 4 + (4 if case["grad"] else 0)) + weights * 2 * passes + kept,
                "flops": passes * sum(18.0 * p * a * b for p, a, b in convs)}
    px = case["images"] * case["rows"] * case["cols"]
    ci, co = case["cin"], case["cout"]
    return {"bytes": px * 2 * (ci + co) * 2 + 9 * ci * co * (2 + 2 + 4),
            "flops": 3 * 18.0 * px * ci * co}


# --------------------------------------------------------------------------
# The step in 64 bits: the weighted cellular automaton of the reference
# (src/kernels/physics.h, src/common/model.c), whole-array torch.

LAND, SEA, WALL = 0, 1, 2


class _Exact:
    def __init__(self, f, K):
        self.p = p = f["p"]
        self.K = K
        d = lambda t: t.to(F64)  # noqa: E731
        self.z, self.n, self.h = d(f["z"]), d(f["n"]).clamp_min(1e-12), d(f["h"]).clone()
        self.cr = d(f["C"]) * d(f["R"])
        m = f["mask"]
        self.land, self.sea, self.wall = m == LAND, m == SEA, m == WALL
        self.all_land = bool(self.land.all())
        self.hmax, self.A = self.h.clone(), DX * DX
        self.width = DX if K == 4 else (math.sqrt(2.0) - 1.0) * DX
        pair = (slice(None, -1), slice(1, None))
        full, a, b = slice(None), pair[0], pair[1]
        # (first cell, second cell, distance) of every face family
        self.fam = [((full, a), (full, b), DX), ((a, full), (b, full), DX)]
        if K == 8:
            dd = math.sqrt(2.0) * DX
            self.fam += [((a, a), (b, b), dd), ((a, b), (b, a), dd)]
        nr, nc = m.shape
        self.sides = []
        if p.boundary == "open":
            for on, sl in zip(p.edges, ((0, full), (nr - 1, full), (full, 0), (full, nc - 1))):
                if on:
                    self.sides.append(sl)

    def level(self):
        if self.all_land:
            return self.z + self.h
        return torch.where(self.sea, torch.full_like(self.z, self.p.z_sea), self.z + self.h)

    def flux(self, dL, hf, nf, S, adL, dt, dead):
        p = self.p
        v = hf.clamp_min(1e-30).pow(2.0 / 3.0) / nf * S.sqrt()
        v = torch.minimum(v, (p.g * hf.clamp_min(0.0)).sqrt())
        q = torch.minimum(v * hf * self.width, adL * self.A / (2 * self.K * dt))
        q = torch.where(dL > 0, q, -q)
        return torch.where(dead | (adL < p.tau_l) | (hf < p.tau_h), torch.zeros_like(q), q)

    def velocity(self):
        """The largest stable velocity over wet LAND cells."""
        p, L = self.p, self.level()
        S = torch.zeros_like(L)
        for a, b, d in self.fam:
            s = (L[a] - L[b]).abs() / d
            if not self.all_land:
                s = torch.where(self.wall[a] | self.wall[b], torch.zeros_like(s), s)
            S[a] = torch.maximum(S[a], s)
            S[b] = torch.maximum(S[b], s)
        for sl in self.sides:
            S[sl] = torch.maximum(S[sl], (L[sl] - (self.z[sl] - p.S_bnd * DX)).abs() / DX)
        v = self.h.clamp_min(1e-30).pow(2.0 / 3.0) / self.n * S.sqrt()
        v = torch.minimum(v, (p.g * self.h).sqrt()).clamp_min(1e-6)
        return float(torch.where(self.land & (self.h >= p.tau_h), v, torch.zeros_like(v)).max())

    def rain(self, t, dt):
        p = self.p
        if p.rain_end > 0 and p.rain_end - t < 1e-9:
            return 0.0
        if p.hyeto == "uniform":
            return dt / 86400.0
        T = p.D_h * 3600.0
        tp = p.phi * T
        f = lambda x: 2 / T * (x / tp if x < tp else (T - x) / (T - tp)) if 0 <= x < T else 0.0  # noqa: E731
        e = min(t + dt, T)
        cuts = [t] + ([tp] if t < tp < e else []) + [e]
        return sum(0.5 * (f(x) + f(y)) * (y - x) for x, y in zip(cuts, cuts[1:])) if t < T else 0.0

    def inflow(self, t, dt):
        p = self.p
        q = lambda x: (0.0 if x <= 0 or x >= p.inflow_t_end else  # noqa: E731
                       p.inflow_peak * (x / p.inflow_t_peak if x <= p.inflow_t_peak else
                                        (p.inflow_t_end - x) / (p.inflow_t_end - p.inflow_t_peak)))
        e = min(t + dt, p.inflow_t_end)
        cuts = [t] + ([p.inflow_t_peak] if t < p.inflow_t_peak < e else []) + [e]
        return sum(0.5 * (q(x) + q(y)) * (y - x) for x, y in zip(cuts, cuts[1:]) if y > x)

    def run(self, steps):
        p, t = self.p, 0.0
        for _ in range(steps):
            v = self.velocity()
            dt = min(p.dt_max, p.alpha * DX / v) if v > 0 else p.dt_max
            dt = max(dt, p.dt_min)
            ends = [p.T_sim]
            for every in (86400.0, p.out_every):
                if every > 0:
                    e = (math.floor(t / every) + 1.0) * every
                    ends.append(e + every if e - t < 1e-9 else e)
            if p.rain_end > 0 and p.rain_end - t >= 1e-9:
                ends.append(p.rain_end)
            hit = min(ends) - t <= dt
            if hit:
                dt = min(ends) - t
            F, Vin = self.rain(t, dt), self.inflow(t, dt)
            self.step(dt, F, Vin)
            t = min(ends) if hit else t + dt

    def step(self, dt, F, Vin):
        p, L = self.p, self.level()
        ze = self.z if self.all_land else torch.where(self.sea, torch.full_like(self.z, p.z_sea),
                                                      self.z)
        out = torch.zeros_like(L)
        qs = []
        for a, b, d in self.fam:
            dL = L[a] - L[b]
            adL = dL.abs()
            hf = torch.maximum(L[a], L[b]) - torch.maximum(ze[a], ze[b])
            nf = 0.5 * (self.n[a] + self.n[b])
            dead = torch.zeros_like(dL, dtype=torch.bool)
            if not self.all_land:
                sa, sb = self.sea[a], self.sea[b]
                nf = torch.where(sa, self.n[b], torch.where(sb, self.n[a], nf))
                dead = self.wall[a] | self.wall[b] | torch.where(dL > 0, sa, sb)
            q = self.flux(dL, hf, nf, adL / d, adL, dt, dead)
            out[a] += q.clamp_min(0.0)
            out[b] += (-q).clamp_min(0.0)
            qs.append(q)
        qo = []
        for sl in self.sides:
            lo = self.z[sl] - p.S_bnd * DX
            dL = L[sl] - lo
            hf = torch.maximum(L[sl], lo) - torch.maximum(self.z[sl], lo)
            q = self.flux(dL, hf, self.n[sl], dL.abs() / DX, dL.abs(), dt, ~self.land[sl])
            qo.append(q.clamp_min(0.0))
            out[sl] += qo[-1]
        ov, hold = out * dt, self.h * self.A
        s = torch.where(self.land & (ov > hold) & (ov > 0), hold / ov.clamp_min(1e-300),
                        torch.ones_like(ov))
        net = torch.zeros_like(L)
        for (a, b, _), q in zip(self.fam, qs):
            q = q * torch.where(q >= 0, s[a], s[b])
            net[a] -= q
            net[b] += q
        for sl, q in zip(self.sides, qo):
            net[sl] -= q * s[sl]
        h = (self.h + (dt * (net / self.A) + self.cr * F)).clamp_min(0.0)
        if p.inflow_cell >= 0:
            r, c = divmod(p.inflow_cell, h.shape[1])
            h[r, c] += Vin / self.A
        self.h = torch.where(self.land, h, self.h)
        self.hmax = torch.where(self.land, torch.maximum(self.hmax, self.h), self.hmax)


def _exact_ca(case, seed):
    e = _Exact(_scenario(case, seed), case["K"])
    e.run(case["steps"])
    return e


def _conv64(x, w):
    """[N, H, W, C] with [co, 9, ci] weights, padding 1, as nine products."""
    N, H, W, ci = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    y = 0.0
    for k in range(9):
        y = y + xp[:, k // 3:k // 3 + H, k % 3:k % 3 + W] @ w[:, k].T
    return y


def _exact_unet(case, seed):
    """The network on the model's rounded weights with no other rounding."""
    x, _ = _images(case, seed)
    model = UNet(seed=seed % 1000)
    ws = [(c.w.to(torch.bfloat16).to(F64), c.b.to(F64)) for c in model.convs()]
    hw, hb = model.hw.to(F64), model.hb.to(F64)
    out = []
    for xi in x.to(torch.bfloat16).to(F64).split(4):
        conv = lambda a, i: (_conv64(a, ws[i][0]) + ws[i][1]).clamp_min(0.0)  # noqa: E731
        cur = torch.nn.functional.pad(xi, (0, ws[0][0].shape[2] - 4))
        skips = []
        for lvl in range(4):
            cur = conv(conv(cur, 2 * lvl), 2 * lvl + 1)
            if lvl < 3:
                skips.append(cur)
                N, H, W, ch = cur.shape
                cur = cur.view(N, H // 2, 2, W // 2, 2, ch).amax((2, 4))
        for j in range(3):
            up = cur.repeat_interleave(2, 1).repeat_interleave(2, 2)
            cur = conv(conv(torch.cat([up, skips[2 - j]], -1), 8 + 2 * j), 9 + 2 * j)
        out.append(cur @ hw + hb)
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ca":
        e = _exact_ca(case, seed)
        # the time of the peak jumps between steps where a depth barely rises
        return {"h": e.h, "hmax": e.hmax, "tmax": None}
    if kind == "dropin":
        e = _Exact(_dropin_fields(case, seed), 4)
        e.run(case["steps"])
        return {"h": e.h, "hmax": e.hmax, "tmax": None, "steps": None}
    if kind == "batch":
        got = [_exact_ca(c, s) for c, s in _batch_cases(case, seed)]
        return {"h": [e.h for e in got], "hmax": [e.hmax for e in got]}
    if kind == "unet":
        if case["mc"] or case["grad"]:
            return None        # the dropout mask is the library's own hash
        return {"out": _exact_unet(case, seed)}
    x, dy, w, b = (t.to(F64) for t in _conv_inputs(case, seed))
    pad = lambda t: torch.nn.functional.pad(t, (0, 0, 1, 1, 1, 1))  # noqa: E731
    y = pad((_conv64(x, w) + b).clamp_min(0.0))
    dx = pad(_conv64(dy, w.flip(1).permute(2, 1, 0)))
    N, H, W, ci = x.shape
    xp = pad(x)
    dw = torch.stack([torch.einsum("nhwo,nhwi->oi", dy,
                                   xp[:, k // 3:k // 3 + H, k % 3:k % 3 + W]) for k in range(9)], 1)
    return {"y": y.flatten(0, 2), "dx": dx.flatten(0, 2), "dw": dw}

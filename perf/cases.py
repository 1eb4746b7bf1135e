"""What a user of this framework has it compute, as measurable cases.

Every case is one pass through the public entry points: a coupled step of one
domain (`Model.advance`), of a ragged batch (`Batch.advance`), or the wave
surrogate's inference and training step (`UNet.forward`, `UNet.train_step`).
The states are made on the GPU from the seed: a sloping beach with a bar, a
shoaling and breaking directional sea with rollers, long waves, currents and
suspended sediment, as a run meets them some minutes after its start.

`exact` restates one coupled step (and the network) in 64-bit torch, so that
the rounding of the framework's results can be measured against it.
"""
import math

import numpy as np
import torch

from xbeach_gpu_b200.abi import XBG_FP32, XBG_FP64, default_params, sanity
from xbeach_gpu_b200.model import Batch, Model
from xbeach_gpu_b200.surrogate import IN_CH, OUT_CH, UNet

PI = 3.14159265
DEV = "cuda"


def listed():
    return [
        # the reference's CPU-runnable beach (200 x 100, 10 bins): the smallest
        # run a user makes, four steps per call
        dict(name="beach_200x100", kind="step", nx=200, ny=100, nt=10, span=50, dx=5.0, hmax=10.0, slope=0.02,
             bar=0, Hs=1.5, Tp=10.0, morfac=1.0, steps=4),
        # a grid of odd sides, as surveyed areas give them (rows not 16-byte aligned)
        dict(name="odd_509x251", kind="step", nx=509, ny=251, nt=12, span=90, dx=4.0, hmax=12.0, slope=0.025,
             bar=1, Hs=2.0, Tp=9.0, morfac=1.0, steps=2),
        # an ordinary site model: barred beach, 18 bins, bed update accelerated
        dict(name="barred_1024x512", kind="step", nx=1024, ny=512, nt=18, span=90, dx=2.0, hmax=15.0, slope=0.025,
             bar=1, Hs=2.5, Tp=12.0, morfac=10.0, steps=2),
        # the large single domain of the benchmark
        dict(name="barred_2048x1024", kind="step", nx=2048, ny=1024, nt=18, span=90, dx=2.0, hmax=15.0, slope=0.025,
             bar=1, Hs=2.5, Tp=12.0, morfac=10.0, steps=2),
        # wave-current interaction on (rip and tidal currents act on the waves)
        dict(name="wci_768x384", kind="step", nx=768, ny=384, nt=12, span=60, dx=4.0, hmax=12.0, slope=0.02,
             bar=1, Hs=2.0, Tp=10.0, morfac=1.0, wci=1, steps=2),
        # waves and flow only: Baldock breaking, no roller, fixed bed
        dict(name="hydro_1280x640", kind="step", nx=1280, ny=640, nt=9, span=45, dx=4.0, hmax=20.0, slope=0.02,
             bar=0, Hs=3.0, Tp=13.0, sed=0, roller=0, breakmodel=2, steps=2),
        # flow alone (surge and long waves without the wave solver)
        dict(name="flow_1536x768", kind="step", nx=1536, ny=768, nt=1, span=90, dx=5.0, hmax=20.0, slope=0.02,
             bar=0, Hs=0.0, Tp=10.0, swave=0, sed=0, steps=2),
        # the double-precision build
        dict(name="fp64_512x256", kind="step", nx=512, ny=256, nt=18, span=90, dx=2.0, hmax=15.0, slope=0.025,
             bar=1, Hs=2.5, Tp=12.0, morfac=10.0, fp64=1, steps=2),
        # a ragged ensemble: each scenario with its own grid, slope, sea and dt
        dict(name="ensemble_10", kind="batch", n=10, nxlo=128, nxhi=1024, nylo=64, nyhi=512, nt=12, pick=3, steps=2),
        # the wave surrogate predicting one 1024 x 512 domain
        dict(name="surrogate_512x1024", kind="infer", B=1, H=512, W=1024, base=32),
        # the surrogate's training step on a batch of crops
        dict(name="surrogate_train_4x256", kind="train", B=4, H=256, W=256, base=32),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["step"] * 9 + ["batch"] * 2 + ["infer", "train"])
    if kind == "infer":
        return dict(kind="infer", B=1, H=8 * logint(16, 64), W=8 * logint(16, 128), base=32)
    if kind == "train":
        return dict(kind="train", B=rng.choice([1, 2, 4]), H=16 * logint(6, 16), W=16 * logint(6, 16), base=32)
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(4, 10), nxlo=128, nxhi=1024, nylo=64, nyhi=512,
                    nt=rng.choice([8, 10, 12, 18]), pick=rng.randrange(1 << 20), steps=2)
    c = dict(kind="step", nx=logint(160, 2048), ny=logint(80, 1024), nt=rng.choice([6, 8, 9, 10, 12, 15, 18, 24]),
             span=rng.choice([45, 60, 90]), dx=rng.choice([2.0, 4.0, 5.0]), hmax=round(rng.uniform(8.0, 20.0), 1),
             slope=round(rng.uniform(0.012, 0.045), 4), bar=rng.choice([0, 1]), Hs=round(rng.uniform(0.5, 4.0), 2),
             Tp=round(rng.uniform(6.0, 14.0), 1), morfac=rng.choice([1.0, 10.0]), steps=2)
    # most grids have sides in multiples of 4 or 32, the rest are ragged
    m = rng.choice([1, 4, 32])
    c["nx"], c["ny"] = max(160, c["nx"] // m * m), max(80, c["ny"] // m * m)
    option = rng.choice(["", "", "", "", "wci", "noroller", "baldock", "hydro", "flow", "fp64"])
    if option == "wci":
        c["wci"] = 1
    if option == "noroller":
        c["roller"] = 0
    if option == "baldock":
        c["breakmodel"] = 2
    if option == "hydro":
        c["sed"] = 0
    if option == "flow":
        c.update(swave=0, sed=0, nt=1, span=90)
    if option == "fp64":
        c["fp64"] = 1
    most = 2048 * 1024 * 18 // (4 if option in ("wci", "fp64") else 1)
    while c["nx"] * c["ny"] * c["nt"] > most:
        c["nx"], c["ny"] = max(160, c["nx"] * 3 // 4 // m * m), max(80, c["ny"] * 3 // 4 // m * m)
    return c


# ------------------------------------------------------------------ inputs
def _params(c):
    """The parameters of a step case (one scenario of a batch)."""
    p = default_params()
    p.nx, p.ny, p.dx = c["nx"], c["ny"], c["dx"]
    p.swave, p.flow, p.sedtrans, p.morphology = c.get("swave", 1), 1, c.get("sed", 1), c.get("sed", 1)
    p.thetamin, p.thetamax = -c["span"] * PI / 180, c["span"] * PI / 180
    p.dtheta = (p.thetamax - p.thetamin) / c["nt"]
    p.breakmodel, p.roller = c.get("breakmodel", 1), c.get("roller", 1)
    p.wci, p.hwci = float(c.get("wci", 0)), 0.5
    p.D50, p.D90 = c.get("D50", 0.00025), 1.5 * c.get("D50", 0.00025)
    p.morfac, p.sedstart = c.get("morfac", 1.0), 0.0
    p.CFL, p.eps = 0.7, 0.01
    p.wavebndtype, p.dtbc = 4, 2.0
    p.rtlength = 9600.0 if c["nx"] * c["ny"] < 200000 else 2400.0
    p.endtime = 1.0e6
    return sanity(p, 1e9)


def _boundary(c, p, seed):
    """Offshore records St[nrec][nt][ny] and q[nrec][4][ny]: a directional sea
    in seeded wave groups with its bound long wave."""
    rng = np.random.default_rng(seed + 17)
    nt, ny, nrec = p.ntheta, p.ny, int(p.rtlength / p.dtbc) + 2
    theta = p.thetamin + (np.arange(nt) + 0.5) * p.dtheta
    spread = np.cos((theta - c.get("mdir", 0.15)) / 2.0) ** 20
    Sd = spread / spread.sum() * (c["Hs"] ** 2 * p.rho * p.g / (16.0 * p.dtheta))
    t, y = np.arange(nrec) * p.dtbc, np.arange(ny) * p.dx
    w = 2 * math.pi * rng.uniform(0.5, 1.5, 4) / (8.0 * c["Tp"])
    k, a = rng.uniform(-1, 1, 4) * 2 * math.pi / (ny * p.dx), rng.uniform(0, 2 * math.pi, 4)
    env = np.zeros((nrec, ny))
    for j in range(4):
        ct, st = np.cos(w[j] * t + a[j]), np.sin(w[j] * t + a[j])
        env += ct[:, None] * np.cos(k[j] * y) - st[:, None] * np.sin(k[j] * y)
    env = np.clip(1.0 + 0.3 * env, 0.05, None)
    St = env[:, None, :] * Sd[None, :, None]
    q = np.zeros((nrec, 4, ny))
    q[:, 0], q[:, 1] = 0.02 * c["Hs"] * (env - 1.0), 0.005 * c["Hs"] * (env - 1.0)
    return St, q


def _at(a, dx=0, dy=0):
    """a at the neighbour (dx, dy), clamped at the grid's edges."""
    if dx:
        a = a.index_select(-1, (torch.arange(a.shape[-1], device=a.device) + dx).clamp(0, a.shape[-1] - 1))
    if dy:
        a = a.index_select(-2, (torch.arange(a.shape[-2], device=a.device) + dy).clamp(0, a.shape[-2] - 1))
    return a


# every field the state below sets; the other fields of a model start as it makes them
SET = ("zb zs hh uu vv hu hv hum hvm qx qy ueu vev vmageu vmagev vu uv uuold vvold zsold H E D DR R k c cg Fx Fy "
       "urms ust thetamean cfm fwm C stdep umeanbnd ee rr").split()


def _sea(c, p, seed):
    """The fields of a running model, in the element type of the case."""
    R = torch.float64 if c.get("fp64") else torch.float32
    nx, ny, nt = p.nx, p.ny, p.ntheta
    rng = np.random.default_rng(seed + 5)
    g = torch.Generator(device=DEV).manual_seed(seed + 11)
    x = torch.arange(nx, device=DEV, dtype=torch.float64)[None, :] * p.dx
    y = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None] * p.dx

    def smooth():   # long waves over the domain, of order one
        f = torch.zeros(ny, nx, device=DEV, dtype=torch.float64)
        for _ in range(5):
            kx, ky, a = rng.uniform(1, 9) / (nx * p.dx), rng.uniform(-4, 4) / (ny * p.dx), rng.uniform(0, 2 * math.pi)
            f += torch.sin(2 * math.pi * (kx * x + ky * y) + a)
        return 0.45 * f

    f = {}
    xw = 0.8 * nx * p.dx
    zb = torch.clamp((xw - x) * c["slope"], -3.0, c["hmax"]) + 0 * y
    if c["bar"]:
        crest = xw - 0.12 * xw
        zb = zb - (1.0 + 0.4 * torch.sin(2 * math.pi * y / 250.0)) * torch.exp(-(((x - crest) / 40.0) ** 2) / 2)
    f["zb"] = zb + 0.03 * torch.randn(ny, nx, generator=g, device=DEV, dtype=torch.float64)
    f["zs"] = torch.maximum(0.12 * smooth(), -f["zb"])
    f["hh"] = torch.clamp(f["zb"] + f["zs"], min=p.eps)
    hh = f["hh"]
    wet = hh > 2 * p.eps
    surf = torch.clamp(c["Hs"] / hh, max=1.0) * wet
    f["uu"], f["vv"] = 0.25 * smooth() * wet, (0.1 + 0.5 * surf) * smooth() * wet
    f["hu"], f["hv"] = torch.minimum(hh, _at(hh, 1)), torch.minimum(hh, _at(hh, 0, 1))
    f["hum"], f["hvm"] = 0.5 * (hh + _at(hh, 1)), 0.5 * (hh + _at(hh, 0, 1))
    f["qx"], f["qy"] = f["uu"] * f["hu"], f["vv"] * f["hv"]
    f["uuold"], f["vvold"] = f["uu"] + 0.01 * smooth() * wet, f["vv"] + 0.01 * smooth() * wet
    f["zsold"] = f["zs"] + 0.005 * smooth() * wet
    f["vu"], f["uv"] = 0.9 * f["vv"], 0.9 * f["uu"]
    f["ueu"], f["vev"] = f["uu"] - 0.05 * surf, f["vv"] * 0.98
    f["vmageu"], f["vmagev"] = torch.hypot(f["ueu"], f["vu"]), torch.hypot(f["uv"], f["vev"])
    kd = 2 * math.pi / (c["Tp"] * torch.sqrt(p.g * hh))
    f["c"] = torch.sqrt(p.g * hh * torch.tanh(kd * hh).clamp(min=1e-3) / (kd * hh).clamp(min=1e-3)) + 0.05
    f["k"], f["cg"] = 2 * math.pi / (f["c"] * c["Tp"]), 0.9 * f["c"]
    H = torch.minimum(c["Hs"] / math.sqrt(2) * (1 + 0.15 * smooth()).clamp(min=0.2), 0.5 * hh) * wet
    f["H"], f["E"] = H, p.rho * p.g * H ** 2 / 8
    theta = torch.tensor([p.thetamin + (i + 0.5) * p.dtheta for i in range(nt)], device=DEV, dtype=torch.float64)
    sp = torch.cos((theta - c.get("mdir", 0.15)) / 2) ** 20
    sp = sp / sp.sum()
    ripple, phase = smooth(), rng.uniform(0, 2 * math.pi, nt)
    breaking = (H > 0.4 * hh) * 0.15 + 0.002
    f["ee"] = torch.empty(nt, ny, nx, device=DEV, dtype=R)
    f["rr"] = torch.empty(nt, ny, nx, device=DEV, dtype=R)
    for i in range(nt):
        e = f["E"] / p.dtheta * sp[i] * (1 + 0.2 * torch.sin(3 * ripple + phase[i]))
        f["ee"][i], f["rr"][i] = e, e * breaking * torch.sqrt(hh)
    f["R"] = f["rr"].sum(0) * p.dtheta
    f["DR"] = 2 * p.g * p.beta * f["R"] / f["c"]
    f["D"] = f["DR"] * (1 + 0.1 * smooth())
    f["Fx"], f["Fy"] = f["DR"] / f["c"], 0.1 * f["DR"] / f["c"]
    f["urms"] = math.pi * H / c["Tp"] / torch.sinh((f["k"] * hh).clamp(0.05, 10.0)) / math.sqrt(2)
    f["ust"] = (f["E"] + 2 * f["R"]) / f["c"] / p.rho / hh.clamp(min=0.2)
    f["thetamean"] = 0.15 + 0.1 * smooth()
    f["cfm"], f["fwm"] = torch.full_like(hh, p.cfsand), torch.full_like(hh, p.fwsand)
    f["C"] = 1e-3 * surf * (1 + 0.3 * smooth()).clamp(min=0.0)
    f["stdep"] = 5.0 + 0.2 * smooth()
    f["umeanbnd"] = torch.full((ny,), 0.01, device=DEV, dtype=torch.float64)
    return {n: f[n].to(R).contiguous() for n in SET}


def _clock(c, p, f):
    """(time, dt): some minutes into the run, at the time step of the flow."""
    return 300.0, 0.5 * p.CFL * p.dx / math.sqrt(9.81 * float(f["hh"].max()))


LEVEL = ([0.0, 1e7], [0.05, 0.05], [0.10, 0.10])     # sea level at the two lateral ends
WIND = ([0.0, 1e7], [3.0, 3.0], [2.0, 2.0])


class _DeviceArray:
    """A device pointer of a model as an array (the CUDA array interface);
    owner: the object that frees the memory, kept as long as the array."""

    def __init__(self, ptr, shape, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=kind, version=3)


def _view(m, name, owner):
    ptr, n = m.device_ptr(name)
    return torch.as_tensor(_DeviceArray(ptr, (n,), "<f4" if m.dtype == np.float32 else "<f8", owner), device=DEV)


def _fill(m, c, p, seed):
    """Give a model its boundaries, state and clock."""
    St, q = _boundary(c, p, seed)
    m.set_wave_boundary(0, St, q, t0=0.0, tend=p.rtlength, Trep=c["Tp"] / 1.1)
    m.set_sealevel(*LEVEL)
    m.set_wind(*WIND)
    f = _sea(c, p, seed)
    t, dt = _clock(c, p, f)
    m.set_time(t, dt, dt)
    for n in SET:
        v = _view(m, n, m)
        v.copy_(f[n].reshape(-1))
    torch.cuda.synchronize()


# what a user reads of a model after a step
READ = ("zb zs hh uu vv hu hv qx qy ueu vev vu uv vmageu vmagev H E D DR R Fx Fy urms ust thetamean k c cg C ceqsg "
        "stdep dzb dzsdt rolthick Hmean uumean vvmean hhmean zsmean Cmean zsmax").split()


def _names(c):
    names = list(READ)
    if not c.get("swave", 1):
        names = [n for n in names if n not in "H E D DR R Fx Fy urms ust thetamean k c cg Hmean".split()]
    if not c.get("sed", 1):
        names = [n for n in names if n not in "C ceqsg stdep dzb rolthick Cmean zb".split()]
    return names


def _scenarios(c):
    """The scenarios of a batch case, as step cases."""
    rng = np.random.default_rng(c["pick"])
    out = []
    for _ in range(c["n"]):
        out.append(dict(kind="step", nx=32 * int(rng.integers(c["nxlo"] // 32, c["nxhi"] // 32 + 1)),
                        ny=32 * int(rng.integers(c["nylo"] // 32, c["nyhi"] // 32 + 1)), nt=c["nt"], span=90, dx=4.0,
                        hmax=12.0, slope=float(rng.uniform(0.01, 0.05)), bar=int(rng.random() < 0.5),
                        Hs=float(rng.uniform(0.5, 4.0)), Tp=float(rng.uniform(6.0, 14.0)),
                        mdir=float(rng.uniform(-0.5, 0.5)), D50=float(rng.uniform(0.00015, 0.0004)), morfac=1.0,
                        steps=c["steps"]))
    return out


BATCH_READ = "ee rr zs uu vv zb".split()


# ------------------------------------------------------------------ surrogate
def _layers(base):
    c1, c2, c3, c4 = base, 2 * base, 4 * base, 8 * base
    return {"e1a": (IN_CH, c1), "e1b": (c1, c1), "e2a": (c1, c2), "e2b": (c2, c2), "e3a": (c2, c3), "e3b": (c3, c3),
            "e4a": (c3, c4), "e4b": (c4, c4), "d3a": (c4 + c3, c3), "d3b": (c3, c3), "d2a": (c3 + c2, c2),
            "d2b": (c2, c2), "d1a": (c2 + c1, c1), "d1b": (c1, c1), "head": (c1, OUT_CH)}


def _weights(c, seed):
    """Layer weights [cout, 3, 3, cin] and biases, and the normalised input
    planes [B*H*W, IN_CH] with the targets."""
    g = torch.Generator(device=DEV).manual_seed(seed + 3)
    W = {}
    for n, (ci, co) in _layers(c["base"]).items():
        gain = 1.0 if n == "head" else 2.0
        W[n] = (torch.randn(co, 3, 3, ci, generator=g, device=DEV) * math.sqrt(gain / (9 * ci)),
                0.02 * torch.randn(co, generator=g, device=DEV))
    P = c["B"] * c["H"] * c["W"]
    x = torch.randn(P, IN_CH, generator=g, device=DEV)
    x[:, -2:] = 0
    tgt = 0.5 * torch.randn(P, OUT_CH, generator=g, device=DEV)
    return W, x.to(torch.bfloat16), tgt


def _net(c, W, seed):
    net = UNet(seed=0, base=c["base"])
    for n, (w, b) in W.items():
        l = net.L[n]
        l.w.zero_()
        l.w[:w.shape[0], :w[0].numel()] = w.reshape(w.shape[0], -1)
        l.b.zero_()
        l.b[:b.shape[0]] = b
        l.sync_copies()
    return net


# ------------------------------------------------------------------ the case functions
def prepare(case, seed):
    c = case
    if c["kind"] in ("infer", "train"):
        W, x, tgt = _weights(c, seed)
        return dict(case=c, net=_net(c, W, seed), x=x, tgt=tgt)
    if c["kind"] == "batch":
        sc = _scenarios(c)
        ps = [_params(s) for s in sc]
        b = Batch(ps)
        for k, (s, p) in enumerate(zip(sc, ps)):
            _fill(b.scenario(k), s, p, seed + 101 * k)
        ms = [b.scenario(k) for k in range(c["n"])]
    else:
        p = _params(c)
        b = Model(p, XBG_FP64 if c.get("fp64") else XBG_FP32)
        _fill(b, c, p, seed)
        ms = [b]
    return dict(case=c, model=b, out=_outputs(c, ms, b))


def _outputs(c, ms, owner):
    """The output fields of the models, in place on the device.  A pass is an
    even number of steps, after which ee and rr are in the buffers they were in
    before it."""
    names = BATCH_READ if c["kind"] == "batch" else _names(c) + (["ee", "rr"] if c.get("swave", 1) else [])
    return [{n: _view(m, n, owner) for n in names} for m in ms]


def run(state):
    c = state["case"]
    if c["kind"] == "infer":
        return dict(out=state["net"].forward(state["x"], c["B"], c["H"], c["W"]))
    if c["kind"] == "train":
        net = state["net"]
        loss = net.train_step(state["x"], state["tgt"], c["B"], c["H"], c["W"])
        return dict(loss=loss, **{n: (l.w, l.b, l.gw, l.gb) for n, l in net.L.items()})
    state["model"].advance(c["steps"])
    return state["out"]


def work(case):
    c = case
    if c["kind"] in ("infer", "train"):
        H, W, P, flops, weights, acts = c["H"], c["W"], c["B"] * c["H"] * c["W"], 0, 0, 0
        for n, (ci, co) in _layers(c["base"]).items():
            lvl = {"1": 0, "2": 1, "3": 2, "4": 3}.get(n[1], 0) if n != "head" else 0
            flops += 2 * 9 * ci * co * (P >> (2 * lvl))
            weights += 9 * ci * co + co
        b = P * (IN_CH * 2 + 16 * 4) + 2 * weights
        if c["kind"] == "train":   # weights, gradients and both moments read and written, targets read
            flops, b = 3 * flops, P * (IN_CH * 2 + OUT_CH * 4) + 4 * 7 * weights
        return dict(bytes=b, flops=flops)
    cells = sum(s["nx"] * s["ny"] for s in _scenarios(c)) if c["kind"] == "batch" else c["nx"] * c["ny"]
    # planes a step cannot do without: the persistent fields read and written
    # once, the directional planes too
    swave, sed = c.get("swave", 1), c.get("sed", 1)
    planes = 34 + (26 if swave else 0) + (17 if sed else 0)
    theta = (4 if c.get("roller", 1) else 2) * c["nt"] if swave else 0
    el = 8 if c.get("fp64") else 4
    per_cell = 150 + (120 if sed else 0) + ((400 + 110 * c["nt"]) if swave else 0)
    return dict(bytes=c["steps"] * cells * el * (planes + theta), flops=c["steps"] * cells * per_cell)


# ------------------------------------------------------------------ 64-bit results
def _dispersion(p, sg, h):
    """k, c, cg by the golden-ratio relaxation the model defines."""
    phi = (1 + math.sqrt(5.0)) / 2
    L0 = 2 * math.pi * p.g / sg ** 2
    L1, open_ = torch.full_like(h, L0), torch.ones_like(h, dtype=torch.bool)
    for _ in range(198):
        L2 = L0 * torch.tanh(2 * PI * h / L1)
        L1 = torch.where(open_, (L1 + phi * L2) / (phi + 1), L1)
        # the error is that of the relaxation before its update
        err = torch.abs(L2 - (L1 * (phi + 1) - phi * L2))
        open_ = open_ & (err > 1e-4)
        if not bool(open_.any()):
            break
    k = 2 * PI / L1
    c = sg / k
    kh = torch.clamp(k * h, max=10.0)
    return k, c, c * (0.5 + kh / torch.sinh(2 * kh)), kh


def _upwind(q, v, vm, d, axis):
    """Second-order upwind flux difference of q along an axis for the face
    speeds v (upper face) and vm (lower face); d = 1 / spacing."""
    a = (lambda n: _at(q, n, 0)) if axis == "x" else (lambda n: _at(q, 0, n))

    def ext(near, far):
        e = 1.5 * near - 0.5 * far
        return torch.where(e < 0, near, e)

    up = torch.where(v > 0, ext(q, a(-1)), ext(a(1), a(2))) * v
    lo = torch.where(vm > 0, ext(a(-1), a(-2)), ext(q, a(1))) * vm
    return (up - lo) * d


def _theta_adv(q, ct, dth):
    nt = q.shape[0]
    if nt == 1:
        return torch.zeros_like(q)
    i = torch.arange(nt, device=q.device)
    n = lambda k: q[(i + k).clamp(0, nt - 1)]   # noqa: E731
    cb = 0.5 * (ct + ct[(i + 1).clamp(max=nt - 1)])

    def ext(near, far):
        e = 1.5 * near - 0.5 * far
        return torch.where(e < 0, near, e)

    f = cb * torch.where(cb > 0, ext(q, n(-1)), ext(n(1), n(2)))
    f[nt - 1] = 0
    return torch.cat([f[:1], f[1:] - f[:-1]]) / dth


def _edge_rows(q, w):
    """The lateral rows take their neighbour rows' values (times w)."""
    q = q.clone()
    a, b = q[..., 1, :].clone(), q[..., -2, :].clone()
    q[..., 0, :], q[..., -1, :] = a * (w[0] if w is not None else 1), b * (w[-1] if w is not None else 1)
    return q


def _wave(p, s, St, t, dt, Trep):
    nt, dth, g, rho = p.ntheta, p.dtheta, p.g, p.rho
    sg = 2 * PI / Trep
    hh, uu, vv = s["hh"], s["uu"], s["vv"]
    th = torch.tensor([i * dth + p.thetamin + 0.5 * dth for i in range(nt)], device=DEV, dtype=torch.float64)
    cx, sx = torch.cos(th)[:, None, None], torch.sin(th)[:, None, None]
    wet = (hh > p.eps).double()
    ee, rr = s["ee"].clone(), s["rr"].clone()
    ee[:, :, 0] = St * min(t / 100.0, 1.0)
    ee = ee.clamp(min=0.0)
    k, c, cg, kh = _dispersion(p, sg, hh)
    wci = p.wci * torch.clamp(hh / p.hwci, max=1.0)
    ny, nx = hh.shape
    spx = torch.full((nx,), 2 * p.dx, device=DEV, dtype=torch.float64)
    spy = torch.full((ny, 1), 2 * p.dx, device=DEV, dtype=torch.float64)
    spx[0] = spx[-1] = spy[0] = spy[-1] = p.dx
    sl = {n: ((_at(a, 1) - _at(a, -1)) / spx, (_at(a, 0, 1) - _at(a, 0, -1)) / spy)
          for n, a in (("h", hh), ("u", uu), ("v", vv))}
    sig = sg / torch.sinh(2 * kh)
    ct = sig * (sl["h"][0] * sx - sl["h"][1] * cx)
    if p.wci:
        ct = ct + wci * (cx * (sx * sl["u"][0] - cx * sl["u"][1]) + sx * (sx * sl["v"][0] - cx * sl["v"][1]))
    ct = ct.clamp(-0.25 * sg, 0.25 * sg)
    s["wavedt"] = float(torch.clamp(p.CFL * dth / ct.abs().amax(0), max=9999999.9).min())

    def advect(q, v):
        for i in range(nt):   # one bin's x and y fluxes at a time
            a, b = float(torch.cos(th[i])), float(torch.sin(th[i]))
            fx = [0.5 * (v * a + uu * wci + _at(v, n) * a + _at(uu, n) * wci) for n in (1, -1)]
            fy = [0.5 * (v * b + vv * wci + _at(v, 0, n) * b + _at(vv, 0, n) * wci) for n in (1, -1)]
            yield _upwind(q[i], fx[0], fx[1], 1 / p.dx, "x") + _upwind(q[i], fy[0], fy[1], 1 / p.dx, "y")

    thadv = _theta_adv(ee, ct, dth)
    ee = torch.stack([ee[i] - dt * (xy + thadv[i]) for i, xy in enumerate(advect(ee, cg))])
    ee = _edge_rows(ee, wet).clamp(min=0.0)
    Ht = torch.sqrt(ee.sum(0) * dth / (rho * g / 8))
    ee = ee / (Ht / (p.gammax * hh)).square().clamp(min=1.0)
    Ht = torch.minimum(Ht, p.gammax * hh)
    E = rho * g * Ht ** 2 / 8
    if p.breakmodel == 1:
        Qb = (1 - torch.exp((-(Ht / p.gammaa / hh) ** p.n).clamp(min=-100.0))).clamp(max=1.0)
        D = Qb * 2 * p.alpha / Trep * E * Ht / hh
    else:
        Hb = 0.88 / k * torch.tanh(p.gammaa * k * hh / 0.88)
        Qb = torch.exp(-(Hb / Ht.clamp(min=1e-5)) ** 2)
        D = 0.25 * p.alpha * Qb * rho / Trep * g * (Hb ** 2 + Ht ** 2)
    uorb = PI * Ht / (Trep * torch.sinh((k * hh).clamp(max=10.0)))
    D = D + 0.66666666 / PI * rho * s["fwm"] * uorb ** 3
    if p.roller == 1:
        thadv = _theta_adv(rr, ct, dth)
        rr = torch.stack([rr[i] - dt * (xy + thadv[i]) for i, xy in enumerate(advect(rr, c))])
        rr = _edge_rows(rr, wet)
    dd = ee * D / E.clamp(min=1e-7)
    speed = torch.sqrt((c * cx + uu * wci) ** 2 + (c * sx + vv * wci) ** 2) if p.wci else c
    rrd = 2 * g * p.beta * rr / speed * wet
    rr = (rr + dt * (dd - rrd)).clamp(min=0.0) * wet
    ee = (ee - dt * dd).clamp(min=0.0) * wet
    ee = _edge_rows(ee, wet)
    sume = ee.sum(0).clamp(min=1e-5)
    s.update(ee=ee, rr=rr, k=k, c=c, cg=cg, D=D, R=rr.sum(0) * dth, DR=rrd.sum(0) * dth, E=sume * dth,
             thetamean=(ee * th[:, None, None]).sum(0) / sume, H=torch.sqrt(sume * dth / (rho * g / 8)))
    n, tot = cg / c, ee.sum(0)
    Sxx = (n * ((1 + cx * cx) * ee).sum(0) - 0.5 * tot) * dth + (cx * cx * rr).sum(0) * dth
    Syy = (n * ((1 + sx * sx) * ee).sum(0) - 0.5 * tot) * dth + (sx * sx * rr).sum(0) * dth
    Sxy = n * (sx * cx * ee).sum(0) * dth + (sx * cx * rr).sum(0) * dth
    Fx = -(_at(Sxx, 1) - Sxx) / p.dx - 0.25 * (_at(Sxy, 0, 1) + _at(Sxy, 1, 1) - _at(Sxy, 0, -1) - _at(Sxy, 1, -1)) / p.dx
    Fy = -(_at(Syy, 0, 1) - Syy) / p.dx - 0.25 * (_at(Sxy, 1) + _at(Sxy, 1, 1) - _at(Sxy, -1) - _at(Sxy, -1, 1)) / p.dx
    hm = hh.clamp(min=0.2)
    cm = c.clamp(min=math.sqrt(0.2 * g))
    s["urms"] = PI * s["H"] / Trep / torch.sinh((k.clamp(min=0.01) * hm).clamp(max=10.0)) / math.sqrt(2.0)
    ust = (s["E"] + 2 * s["R"]) / cm / rho / hm

    def first_column(o, f):
        f = f.clone()
        f[:, 0] = o[:, 1] * wet[:, 0]
        return f

    s["Fx"] = _edge_rows(Fx, wet)
    s["Fy"], s["ust"] = first_column(Fy, _edge_rows(Fy, wet)), first_column(ust, _edge_rows(ust, wet))


def _offshore(p, s, q, t, dt, Trep, frac):
    """The offshore column of the flow (absorbing-generating boundary)."""
    ny = p.ny
    z0, z1 = LEVEL[1][0], LEVEL[2][0]
    zb = z0 + (z1 - z0) * torch.arange(ny, device=DEV, dtype=torch.float64) / ny
    fac = dt / (4.0 * Trep) if p.swave else dt / 60.0
    ui = 0.0
    if p.swave:
        ui = (q[0] + frac * (q[1] - q[0])) * min(t / 100.0, 1.0) / (zb + s["zb"][:, 0])
    zp = s["zs"][:, 1].clone()
    ur = -torch.sqrt(p.g / s["hh"][:, 0]) * (zp - zb)
    s["umeanbnd"] = fac * s["uu"][:, 0].mean() + s["umeanbnd"] * (1 - fac)
    for n in ("uu", "zs", "vv"):
        s[n] = s[n].clone()
    s["uu"][:, 0], s["zs"][:, 0], s["vv"][:, 0] = 2 * ui + ur + s["umeanbnd"], zp, s["vv"][:, 1].clone()


def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a > 0, torch.minimum(a, b), torch.maximum(a, b)), torch.zeros_like(a))


def _inflow(q, jump, fast, slow):
    """One upwind advection term: none without inflow, the bore form where the
    velocity rises steeply, else the conservative form."""
    return torch.where(q > 0, torch.where(jump > 0.5, fast, slow), torch.zeros_like(q))


def _flow(p, s, dt):
    dx, g, rho, eps = p.dx, p.g, p.rho, p.eps
    A = _at
    zs, zb, hh, uu, vv, hu, hv = (s[n] for n in "zs zb hh uu vv hu hv".split())
    col = torch.arange(p.nx, device=DEV)[None, :]
    row = torch.arange(p.ny, device=DEV)[:, None]
    inx, iny = col > 0, row > 0
    hm, hn = 0.5 * (hh + A(hh, 1)), 0.5 * (hh + A(hh, 0, 1))
    wu, wv = ((hu > eps) & (hm > eps)).double(), ((hv > eps) & (hn > eps)).double()
    hum, hvm = hm.clamp(min=eps), hn.clamp(min=eps)
    # u: advection, viscosity, Euler step
    ul, ur, ut, ub = A(uu, -1), A(uu, 1), A(uu, 0, 1), A(uu, 0, -1)
    q = 0.5 * (hu * uu + A(hu, -1) * ul)
    adv = _inflow(q, uu - ul, 0.5 * (ul + uu) * (uu - ul) / dx, q / hum * (uu - ul) / dx)
    q = -0.5 * (hu * uu + A(hu, 1) * ur)
    adv = adv + _inflow(q, ur - uu, -0.5 * (ur + uu) * (uu - ur) / dx, q / hum * (uu - ur) / dx)
    vb, vbr, vr = A(vv, 0, -1), A(vv, 1, -1), A(vv, 1)
    q = 0.5 * (vb * A(hv, 0, -1) + vbr * A(hv, 1, -1))
    adv = adv + _inflow(q, vv - vb, 0.5 * (vb + vbr) * (uu - ub) / dx, q / hum * (uu - ub) / dx)
    q = -0.5 * (vv * hv + vr * A(hv, 1))
    adv = adv + _inflow(q, A(vv, 0, 1) - vv, -0.5 * (vv + vr) * (uu - ut) / dx, q / hum * (uu - ut) / dx)
    turb = p.nuhfac * hh * (s["DR"] / rho) ** (1.0 / 3.0)
    if p.usesmago == 1:
        dudx, dvdy = (uu - ul) / dx, (vv - vb) / dx
        dudy = 0.5 * (ut - ub + A(uu, -1, 1) - A(uu, -1, -1)) / dx
        dvdx = 0.5 * (vr - A(vv, -1) + vbr - A(vv, -1, -1)) / dx
        nu = torch.maximum(p.nuh ** 2 * dx * dx * torch.sqrt(2 * dudx ** 2 + 2 * dvdy ** 2 + (dudy + dvdx) ** 2), turb)
    else:
        nu = turb.clamp(min=p.nuh)
    visc = (A(nu, 1) * A(hh, 1) * (ur - uu) - nu * hh * (uu - ul)) / dx / dx / hum
    nt = 0.25 * (nu + A(nu, 1) + A(nu, 1, 1) + A(nu, 0, 1))
    nb = 0.25 * (nu + A(nu, 1) + A(nu, 1, -1) + A(nu, 0, -1))
    d1 = nt * 0.5 * (hvm + A(hvm, 1)) * (ut - uu) / dx
    d2 = nb * 0.5 * (A(hvm, 0, -1) + A(hvm, 1, -1)) * (uu - ub) / dx
    visc = visc + (d1 - d2) / dx * A(wu, 0, 1) * A(wu, 0, -1) / hum
    wx, wy = WIND[1][0], WIND[2][0]
    tau = s["cfm"] * rho * s["ueu"] * torch.sqrt(1.3456 * s["urms"] ** 2 + s["vmageu"] ** 2)
    un = uu - dt * (adv - visc + g * (A(zs, 1) - zs) / dx + tau / (rho * hu) - s["Fx"] / (rho * hum.clamp(min=0.2)) -
                    1.25 * p.Cd * abs(wx) * wx / (rho * hum) - p.fc * s["vu"])
    us = _edge_rows(torch.where(inx, torch.where(wu > 0, un, torch.zeros_like(un)), uu), None)
    # v, with the new u
    vl, vt = A(vv, -1), A(vv, 0, 1)
    q = 0.5 * (vv * hv + vb * A(hv, 0, -1))
    adv = _inflow(q, vv - vb, 0.5 * (vb - vv) * (vv - vb) / dx, q / hvm * (vv - vb) / dx)
    q = -0.5 * (hv * vv + A(hv, 0, 1) * vt)
    adv = adv + _inflow(q, vt - vv, -0.5 * (vt + vv) * (vv - vt) / dx, q / hvm * (vv - vt) / dx)
    adv = adv * (inx & iny & (row < p.ny - 2))
    usl, uslt, usr, ust = A(us, -1), A(us, -1, 1), A(us, 1), A(us, 0, 1)
    q = 0.5 * (usl * A(hu, -1) + uslt * A(hu, -1, 1))
    adv = adv + _inflow(q, us - usl, 0.5 * (usl + uslt) * (vv - vl) / dx, q / hvm * (vv - vl) / dx)
    q = -0.5 * (us * hu + ust * A(hu, 0, 1))
    adv = adv + _inflow(q, usr - us, -0.5 * (us + usr) * (vv - vr) / dx, q / hvm * (vv - vr) / dx)
    visc = (A(nu, 0, 1) * A(hh, 0, 1) * (vt - vv) - nu * hh * (vv - vb)) / dx / dx / hvm * A(wv, 0, 1) * A(wv, 0, -1)
    nl = 0.25 * (nu + A(nu, -1) + A(nu, -1, 1) + A(nu, 0, 1))
    d1 = nt * 0.5 * (hum + A(hum, 0, 1)) * (vr - vv) / dx
    d2 = nl * 0.5 * (A(hum, -1) + A(hum, -1, 1)) * (vv - vl) / dx
    visc = visc + (d1 - d2) / dx * A(wv, 1) * A(wv, -1) / hvm
    tau = s["cfm"] * rho * s["vev"] * torch.sqrt(1.3456 * s["urms"] ** 2 + s["vmagev"] ** 2)
    vn = vv - dt * (adv - visc + g * (A(zs, 0, 1) - zs) / dx + tau / (rho * hv) - s["Fy"] / (rho * hvm.clamp(min=0.2)) +
                    p.fc * s["uv"] - 1.25 * p.Cd * abs(wy) * wy / (rho * hvm))
    vs = torch.where(inx & (row < p.ny - 2), torch.where(wv > 0, vn, torch.zeros_like(vn)), vv)
    lo, hi = vs[1].clone(), vs[p.ny - 3].clone()
    vs[0], vs[p.ny - 2] = lo, hi
    # second-order corrections with the previous step's velocities and fluxes
    uo, vo, qx, qy = s["uuold"], s["vvold"], s["qx"], s["qy"]

    def depth(x0, x1, y0, y1, z=zs):
        mz = mb = None
        for j in range(y0, y1 + 1):
            for i in range(x0, x1 + 1):
                a, b = A(z, i, j), A(zb, i, j)
                mz, mb = (a, b) if mz is None else (torch.minimum(mz, a), torch.minimum(mb, b))
        return mz + mb > 2 * eps

    def pick(cond, f, pos, neg):
        z = torch.zeros_like(f)
        return torch.where(cond, torch.where(f > 0, pos, torch.where(f < 0, neg, z)), z)

    w1 = pick(inx & depth(-2, 2, 0, 0), qx + A(qx, -1),
              0.5 * _minmod(us - A(uo, -1), A(us, -1) - A(uo, -2)), -0.5 * _minmod(uo - A(us, -1), A(uo, 1) - us))
    w2 = pick(inx & iny & depth(0, 1, -1, 2), A(qy, 1) + qy,
              0.5 * _minmod(A(us, 0, 1) - uo, us - A(uo, 0, -1)),
              -0.5 * _minmod(A(uo, 0, 1) - us, A(uo, 0, 2) - A(us, 0, 1)))
    qe, qw = 0.5 * (A(qx, 1) + qx), 0.5 * (qx + A(qx, -1))
    qn, qs = 0.5 * (A(qy, 0, -1) + A(qy, 1, -1)), 0.5 * (qy + A(qy, -1))
    u = us - torch.where(inx & iny, dt / hum * ((qe * A(w1, 1) - qw * w1) / dx + (qs * w2 - qn * A(w2, 0, -1)) / dx),
                         torch.zeros_like(us))
    low = inx & iny & (row < p.ny - 2)
    w1 = pick(low & depth(0, 0, -2, 2), qy + A(qy, 0, -1),
              0.5 * _minmod(vs - A(vo, 0, -1), A(vs, 0, -1) - A(vo, 0, -2)),
              -0.5 * _minmod(vo - A(vs, 0, -1), A(vo, 0, 1) - vs))
    w2 = pick(low & depth(-1, 2, 0, 1), A(qx, 0, 1) + qx,
              0.5 * _minmod(A(vs, 1) - vo, vs - A(vo, -1)), -0.5 * _minmod(A(vo, 1) - vs, A(vo, 2) - A(vs, 1)))
    qe, qw = 0.5 * (A(qx, 0, 1) + qx), 0.5 * (A(qx, -1) + A(qx, -1, 1))
    qn, qs = 0.5 * (qy + A(qy, 0, -1)), 0.5 * (A(qy, 0, 1) + qy)
    v = vs - torch.where(inx & iny, dt / hvm * ((qe * w2 - qw * A(w2, -1)) / dx + (qs * A(w1, 0, 1) - qn * w1) / dx),
                         torch.zeros_like(vs))

    def face(vel, i, j):
        b = torch.maximum(-zb, -A(zb, i, j))
        still = (torch.maximum(zs, A(zs, i, j)) - b).clamp(min=eps)
        return torch.where(vel > 0, zs - b, torch.where(vel < 0, A(zs, i, j) - b, still)).clamp(min=0.0)

    hu, hv = face(u, 1, 0), face(v, 0, 1)
    qx, qy = u * hu, v * hv
    dz = (A(qx, -1) - qx + A(qy, 0, -1) - qy) / dx
    s["dzsdt"] = torch.where(inx, dz, s["dzsdt"])
    z, zo = torch.where(inx, zs + dz * dt, zs), s["zsold"]
    w1 = pick(inx & depth(-1, 2, 0, 0, z), u, u * 0.5 * _minmod(A(z, 1) - zo, z - A(zo, -1)),
              -u * 0.5 * _minmod(A(zo, 2) - A(z, 1), A(zo, 1) - z))
    w2 = pick(inx & iny & depth(0, 0, -1, 2, z), v, v * 0.5 * _minmod(A(z, 0, 1) - zo, z - A(zo, 0, -1)),
              v * 0.5 * _minmod(A(zo, 0, 2) - A(z, 0, 1), A(zo, 0, 1) - z))
    core = inx & iny
    z = z - torch.where(core, dt * ((w1 - A(w1, -1)) / dx + (w2 - A(w2, 0, -1)) / dx), torch.zeros_like(z))
    qx, qy = torch.where(core, qx + w1, qx), torch.where(core, qy + w2, qy)
    z = _edge_rows(z, None)
    cs, sn = s["ust"] * torch.cos(s["thetamean"]), s["ust"] * torch.sin(s["thetamean"])
    vu = 0.25 * (A(v, 0, -1) + v + A(v, 1, -1) + A(v, 1)) * wu
    uv = 0.25 * (A(u, -1) + u + A(u, -1, 1) + A(u, 0, 1)) * wv
    ue, ve = u - 0.5 * (cs + A(cs, 1)) * wu, vu - 0.5 * (sn + A(sn, 1)) * wu
    uw, vw = uv - 0.5 * (cs + A(cs, 0, 1)) * wv, v - 0.5 * (sn + A(sn, 0, 1)) * wv
    s.update(uu=u, vv=v, hu=hu, hv=hv, qx=qx, qy=qy, zs=z, hh=(zb + z).clamp(min=eps), uuold=u, vvold=v, zsold=z)
    for n, a in (("vu", vu), ("uv", uv), ("ueu", ue), ("vev", vw), ("vmageu", torch.hypot(ue, ve)),
                 ("vmagev", torch.hypot(uw, vw))):
        s[n] = _edge_rows(a, None)


def _sediment(p, s, dt, Trep):
    A, dx, g, rho, eps = _at, p.dx, p.g, p.rho, p.eps
    hh, c, tm = s["hh"], s["c"], s["thetamean"]
    s["rolthick"] = (s["rolthick"] + dt * (s["dzsdt"].abs() - p.beta * c)).clamp(min=0.0)
    drho = (p.rhosed - rho) / rho
    dst = (drho * g) ** (1.0 / 3.0) / 0.0001 * p.D50
    h = hh.clamp(min=0.01)
    speed = (0.5 * (A(s["ueu"], -1) + s["ueu"])) ** 2 + (0.5 * (A(s["vev"], 0, -1) + s["vev"])) ** 2
    ML = torch.minimum(torch.sqrt(2 * s["R"] * Trep / (rho * c)), h).clamp(min=0.01)
    dcf = (1 / (torch.exp(h.clamp(max=100.0) / ML) - 1)).clamp(max=1.0)
    U2 = s["urms"] ** 2 + 1.45 * p.nuhfac * (s["DR"] / rho) ** (2.0 / 3.0) * dcf
    Ts = (0.1 * h / p.wws).clamp(min=0.5)
    Ucr = (0.19 * p.D50 ** 0.1 if p.D50 <= 0.0005 else 8.5 * p.D50 ** 0.6) * torch.log10(4 * h / p.D90)
    Cd = (0.4 / (torch.log(h.clamp(min=0.06) / 0.006) - 1)) ** 2
    Asb = 0.005 * h * (1 / h / (drho * g)) ** 1.2
    Ass = 0.012 * p.D50 * dst ** -0.6 / (drho * g * p.D50) ** 1.2
    T1 = torch.sqrt(torch.minimum(speed + 0.018 / Cd * U2, 100000.0 * g / s["cfm"] * p.D50 * drho))
    wet = (h > eps).double()
    T2 = torch.where((T1 > Ucr) & (h > eps), (T1 - Ucr).clamp(min=0.0) ** 2.4, torch.zeros_like(h))
    ceq = ((Ass * T2 / h).clamp(max=0.05) + (Asb * T2 / h).clamp(max=0.05)) * wet
    s["ceqsg"] = ceq
    k = 2 * PI / (c * Trep)
    Ur = (3.0 / 8.0 * math.sqrt(2.0) * s["H"] * k / (k * hh) ** 3).clamp(min=1e-5)
    m2, m3, m4, m5, m6 = 0.7939, -0.6065, 0.3539, 0.6373, 0.5995
    Bm = m2 / (1 + math.exp(m3 / m4) * Ur ** (-math.log10(math.e) / m4))
    B1 = (-90 + 90 * torch.tanh(m5 / Ur ** m6)) * PI / 180
    ua = (p.facsk * Bm * torch.cos(B1) - p.facas * Bm * torch.sin(B1)) * s["urms"]
    fac = (s["stdep"] / (p.morfac * dt / (1 - p.por) * hh * ceq / Ts).clamp(min=1e-6)).clamp(max=1.0)
    Cc, zb, hu, hv = s["C"], s["zb"], s["hu"], s["hv"]
    ax, ay = 0.5 * (ua + A(ua, 1)), 0.5 * (ua + A(ua, 0, 1))
    cs, sn = torch.cos(tm), torch.sin(tm)
    ur, vr = s["ueu"] + cs * ax, s["vev"] + sn * ay
    mu = torch.hypot(s["uu"] + cs * ax, s["vu"] + sn * ax)
    mv = torch.hypot(s["uv"] + cs * ay, s["vv"] + sn * ay)
    Cr, Ct = A(Cc, 1), A(Cc, 0, 1)
    cu = torch.where(ur > 0, Cc, torch.where(ur < 0, Cr, 0.5 * (Cc + Cr)))
    cv = torch.where(vr > 0, Cc, torch.where(vr < 0, Ct, 0.5 * (Cc + Ct)))
    Dc = p.nuh + p.nuhfac * hh * (s["DR"] / rho) ** (1.0 / 3.0)
    Su = p.sus * (cu * ur * hu - Dc * hu * (Cr - Cc) / dx + 1.6 * cu * mu * hu * (A(zb, 1) - zb) / dx) * (hu > eps)
    Sv = p.sus * (cv * vr * hv - Dc * hv * (Ct - Cc) / dx + 1.6 * cv * mv * hv * (A(zb, 0, 1) - zb) / dx) * (hv > eps)
    ero = fac * hh * ceq / Ts
    q = dt * Ts / (dt + Ts) * (hh * Cc / dt - ((Su - A(Su, -1)) / dx + (Sv - A(Sv, 0, -1)) / dx - ero)) * (hh > eps)
    q = torch.minimum(q.clamp(min=0.0), 0.1 * hh)
    Cn = _edge_rows(q / hh, None)
    Cn[:, 0] = 0
    s["C"] = Cn
    if not p.morfac > 0:
        return

    def copies(a):
        b = _edge_rows(a, None)
        b[:, 0] = a[:, 1]
        return b

    dzg = p.morfac * dt / (1 - p.por) * (ero - q / Ts)
    hh, zb, sd = hh + dzg, copies(zb + dzg), copies(s["stdep"] - dzg)
    most = torch.where(hh > eps, p.wetdzmax, p.drydzmax)

    def slide(zn, sn_):
        d = (zn - zb) / dx
        over, lim = (d.abs() - most) * dx, p.maxslpchg * dt / dx
        up, down = torch.minimum(over.clamp(max=lim), sd), -torch.minimum(over.clamp(max=lim), sn_)
        return torch.where(d.abs() > most, torch.where(d > 0, up, down), torch.zeros_like(d))

    bx, by = slide(A(zb, 1), A(sd, 1)), slide(A(zb, 0, 1), A(sd, 0, 1))
    dd = bx + by
    dd[:, 1:] -= bx[:, :-1]
    dd[1:] -= by[:-1]
    s.update(zb=copies(zb + dd), stdep=copies(sd - dd), zs=s["zs"] - dd, hh=hh - dd, dzb=-dzg - dd)


def _exact_steps(c, seed):
    p = _params(c)
    St, q = (torch.from_numpy(a).to(DEV) for a in _boundary(c, p, seed))
    if not c.get("fp64"):
        St, q = St.float(), q.float()
    s = {n: a.double() for n, a in _sea(c, p, seed).items()}
    t, dt = _clock(c, p, s)
    zero = torch.zeros_like(s["zb"])
    for n in "dzsdt rolthick ceqsg dzb Hmean uumean vvmean hhmean zsmean Cmean zsmax".split():
        s[n] = zero
    Trep = c["Tp"] / 1.1
    s["wavedt"] = 3e38
    for _ in range(c["steps"]):
        wd = dt
        dt = 0.5 * p.CFL * p.dx / math.sqrt(9.81 * float(s["hh"].max()))
        if p.swave:
            dt = min(dt, 0.5 * s["wavedt"])
        if abs(dt - wd) / wd > 0.1:
            dt = wd * (1.1 if dt > wd else 0.9)
        left = min(p.outputtimestep, p.endtime) - t
        dt = left / math.ceil(left / dt)
        t += dt
        r = min(math.floor(t / p.dtbc), St.shape[0] - 2)
        frac = (t - r * p.dtbc) / p.dtbc
        qq = q[r:r + 2, 0].double()
        _offshore(p, s, qq, t, dt, Trep, frac)
        if p.swave:
            a, b = St[r].double(), St[r + 1].double()
            _wave(p, s, a + frac * (b - a), t, dt, Trep)
        _flow(p, s, dt)
        if p.sedtrans:
            _sediment(p, s, dt, Trep)
        for m, n in (("Hmean", "H"), ("uumean", "uu"), ("vvmean", "vv"), ("hhmean", "hh"), ("zsmean", "zs"),
                     ("Cmean", "C")):
            s[m] = s[m] + s[n]
        s["zsmax"] = torch.maximum(s["zsmax"], s["zs"])
    return s


def _exact_net(W, x, c, grad):
    import torch.nn.functional as F
    P = {}
    for n, (w, b) in W.items():
        P[n] = (w.to(torch.bfloat16).double().permute(0, 3, 1, 2).contiguous().requires_grad_(grad),
                b.double().requires_grad_(grad))

    def conv(n, a, relu=True):
        y = F.conv2d(a, P[n][0], P[n][1], padding=1)
        return torch.relu(y) if relu else y

    def up(lo, hi):
        return torch.cat([lo.repeat_interleave(2, 2).repeat_interleave(2, 3), hi], 1)

    a = x.double().reshape(c["B"], c["H"], c["W"], IN_CH).permute(0, 3, 1, 2)
    e1 = conv("e1b", conv("e1a", a))
    e2 = conv("e2b", conv("e2a", F.avg_pool2d(e1, 2)))
    e3 = conv("e3b", conv("e3a", F.avg_pool2d(e2, 2)))
    e4 = conv("e4b", conv("e4a", F.avg_pool2d(e3, 2)))
    d3 = conv("d3b", conv("d3a", up(e4, e3)))
    d2 = conv("d2b", conv("d2a", up(d3, e2)))
    d1 = conv("d1b", conv("d1a", up(d2, e1)))
    out = conv("head", d1, relu=False)
    return P, out.permute(0, 2, 3, 1).reshape(-1, OUT_CH)


def exact(case, seed):
    c = case
    if c["kind"] == "infer":
        W, x, _ = _weights(c, seed)
        with torch.no_grad():
            _, o = _exact_net(W, x, c, False)
        out = torch.zeros(o.shape[0], 16, device=DEV, dtype=torch.float64)
        out[:, :OUT_CH] = o
        return dict(out=out)
    if c["kind"] == "train":
        W, x, tgt = _weights(c, seed)
        P, o = _exact_net(W, x, c, True)
        loss = ((o - tgt.double()) ** 2).mean()
        loss.backward()
        r = dict(loss=loss.detach().reshape(1))
        for n, (w, b) in W.items():
            co, K = w.shape[0], w[0].numel()
            rows, cols = (16 if n == "head" else co), (K + 63) // 64 * 64
            gw, gb, w0, b0 = (torch.zeros(*shape, device=DEV, dtype=torch.float64)
                              for shape in ((rows, cols), (rows,), (rows, cols), (rows,)))
            gw[:co, :K] = P[n][0].grad.permute(0, 2, 3, 1).reshape(co, K)
            gb[:co], w0[:co, :K], b0[:co] = P[n][1].grad, w.double().reshape(co, K), b.double()
            # Adam's first step: the moments' corrections cancel
            r[n] = (w0 - 1e-3 * gw / (gw.abs() + 1e-8), b0 - 1e-3 * gb / (gb.abs() + 1e-8), gw, gb)
        return r
    if c["kind"] == "batch":
        return [{n: s[n].reshape(-1) for n in BATCH_READ}
                for s in (_exact_steps(s, seed + 101 * k) for k, s in enumerate(_scenarios(c)))]
    s = _exact_steps(c, seed)
    names = _names(c) + (["ee", "rr"] if c.get("swave", 1) else [])
    return [{n: s[n].reshape(-1) for n in names}]

"""What the performance of this framework is measured on.

Every case is work that a user has the framework do, through its public entry
points: single depth steps, continuation over many levels, modelling, migration
of one shot and of a batch, linearised (Born) modelling with its adjoint, and
the FWI gradient.  Grids run from 64 x 64 to 512 x 512, on lengths that are
powers of two and on the ragged ones that aperture windows and paddings give.

``listed()`` are the fixed cases, ``draw(rng)`` gives others of the same ranges,
``prepare`` / ``run`` make the inputs and do one pass, ``work`` is the traffic
and arithmetic that a pass cannot do without, and ``exact`` is the same result
in 64 bits by plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pyfwix_b200 import CudaWEM
from pyfwix_b200 import _lib as L
from pyfwix_b200.fwi import FWIGradient
from pyfwix_b200.plan import Plan, sweep

C64, C128, F64 = torch.complex64, torch.complex128, torch.float64
D = 10.0  # grid step in metres, as in the repository's workloads


# ---------------------------------------------------------------- the cases
def _case(name, op, nx, ny, nw, nz, nref, **more):
    c = dict(name=name, op=op, nx=nx, ny=ny, nw=nw, nz=nz, nref=nref, padx=0, pady=0, taper=20, step="pspi",
             eps=0.0, ns=1)
    c.update(more)
    return c


def listed():
    return [
        # one depth step and its adjoint on the smallest grid: the operator inside a
        # user's own depth loop or solver, where launches and latency count
        _case("step-pspi-64", "step", 64, 64, 16, 4, 3, taper=8),
        # the same on a ragged aperture (odd length), NSPS, attenuation on
        _case("step-nsps-105x90", "step", 105, 90, 24, 4, 4, taper=8, step="nsps", eps=0.01),
        # one wavefield continued down through a padded mid-size model, and the adjoint
        # continuation back (Downward.forward, Downward.adjoint)
        _case("downward-200x168", "downward", 180, 150, 40, 6, 4, padx=20, pady=18),
        # plain modelling of one shot with every background field kept (first
        # configuration's grid and band, fewer levels)
        _case("model-128", "model", 128, 128, 64, 24, 4),
        # modelling of two shot groups x two bands on their aperture windows, the model
        # bound anew each pass as in an inversion's loop (Propagator.forward)
        _case("windows-2x2", "windows", 240, 200, 48, 8, 4, ns=2, taper=12),
        # migration of one shot of the batch configuration
        _case("migrate-320", "migrate", 320, 320, 80, 10, 6),
        # four uneven apertures imaged together over four streams; 150, 216 and 270
        # are what shots between the power-of-two grids have
        _case("batch-4-shots", "batch", 270, 270, 64, 6, 6, ns=4),
        # linearised modelling and gradient operator, NSPS, model shared by every
        # frequency (second configuration, fewer levels)
        _case("born-nsps-256", "born", 256, 256, 128, 8, 4, step="nsps"),
        # the same operators on a per-frequency model, PSPI, two shots, odd window
        _case("born-perfreq-135x120", "born", 135, 120, 40, 6, 3, ns=2, taper=12, perfreq=True),
        # FWI gradient, every depth stored (fourth configuration, fewer levels)
        _case("fwi-384", "fwi", 384, 384, 96, 8, 4),
        # FWI gradient with depth checkpoints on a ragged grid with padding
        _case("fwi-checkpoint-250x216", "fwi", 240, 200, 48, 12, 4, padx=10, pady=16, checkpoint=4),
        # the large migration's Born operators, eight references, packed backgrounds
        _case("born-packed-512", "born", 512, 512, 64, 5, 8, rate=16),
    ]


_RANGE = {  # op: (smallest, largest) lateral length, frequencies, levels
    "step": ((48, 512), (8, 64), (2, 4)),
    "downward": ((64, 384), (16, 64), (4, 8)),
    "model": ((64, 384), (24, 96), (8, 24)),
    "windows": ((96, 300), (24, 64), (6, 10)),
    "migrate": ((96, 400), (32, 96), (6, 12)),
    "batch": ((128, 300), (32, 64), (4, 8)),
    "born": ((64, 384), (24, 128), (4, 8)),
    "fwi": ((96, 384), (24, 96), (6, 12)),
}


def _smooth7(n):
    """The smallest length >= n with no prime factor above 7 (what the transforms take)."""
    while True:
        k = n
        for f in (2, 3, 5, 7):
            while k % f == 0:
                k //= f
        if k == 1:
            return n
        n += 1


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    return work(c)["flops"]


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        op = rng.choice(sorted(_RANGE))
        (n0, n1), (w0, w1), (z0, z1) = _RANGE[op]
        nx = _logint(rng, n0, n1)
        # half the draws are square power-of-two-like grids, half any size
        if rng.random() < 0.5:
            nx = min((64, 96, 128, 160, 192, 256, 320, 384, 512), key=lambda m: abs(m - nx))
            nx = min(max(nx, n0), n1)
            ny = nx
        else:
            ny = max(n0, min(n1, int(nx * rng.uniform(0.6, 1.0))))
        # a padded length is one the transforms take
        c = _case("", op, nx, ny, _logint(rng, w0, w1), rng.randint(z0, z1), rng.randint(2, 8),
                  padx=_smooth7(nx) - nx, pady=_smooth7(ny) - ny, taper=rng.choice([0, 8, 12, 20]),
                  step=rng.choice(["pspi", "nsps"]), eps=rng.choice([0.0, 0.0, 0.01]),
                  ns=rng.choice([1, 1, 2]))
        del c["name"]
        if op == "windows":
            c["ns"] = 2
        if op == "batch":
            c["ns"] = rng.randint(2, 4)
        if op == "born":
            # PSPI Born with a taper is not an exact adjoint pair but is what users run
            c["perfreq"] = rng.random() < 0.3
        if op == "fwi":
            c["step"] = "pspi"
            c["nref"] = rng.randint(2, 6)
            if rng.random() < 0.5:
                c["checkpoint"] = rng.choice([2, 3, 4])
        if _cost(c) <= largest:
            return c


# ---------------------------------------------------------------- inputs
def _par(c, **more):
    ow, dw = _band(c)
    p = dict(ox=0.0, oy=0.0, oz=0.0, dx=D, dy=D, dz=D, ow=ow, dw=dw, nref=c["nref"], eps=c["eps"], taperx=c["taper"],
             tapery=c["taper"], padx=c["padx"], pady=c["pady"], step=c["step"], eps_scat=0.04, taylor=1)
    p.update(more)
    return p


def _band(c):
    """3 to 40 Hz over the case's frequencies, at most 1 Hz apart."""
    return 3.0, min(1.0, 37.0 / max(1, c["nw"] - 1))


def _gen(seed, dev):
    return torch.Generator(device=dev).manual_seed(int(seed))


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _velocity(nz, ny, nx, seed):
    """1500 + 0.5 z m/s times a smooth seeded perturbation (+-5 %) and one +10 % body."""
    dev = _dev()
    g = _gen(seed, dev)
    coarse = torch.randn((1, 1, max(2, nz // 4), max(4, ny // 12), max(4, nx // 12)), generator=g, device=dev)
    p = torch.nn.functional.interpolate(coarse, size=(nz, ny, nx), mode="trilinear", align_corners=True)[0, 0]
    p = 0.05 * p / p.abs().max()
    z = D * torch.arange(nz, device=dev)[:, None, None]
    y = torch.arange(ny, device=dev)[None, :, None] / ny
    x = torch.arange(nx, device=dev)[None, None, :] / nx
    c = torch.rand(2, generator=g, device=dev) * 0.5 + 0.25
    body = torch.exp(-(((x - c[0]) / 0.15) ** 2 + ((y - c[1]) / 0.15) ** 2))
    return (1500.0 + 0.5 * z) * (1 + p) * (1 + 0.1 * body)


def _slow2(c, seed):
    """s^2 [nz][ny][nx] float32 on the device."""
    return (1.0 / _velocity(c["nz"], c["ny"], c["nx"], seed) ** 2).float().contiguous()


def _ricker(c, nsrc, seed):
    """[nsrc][nw] spectrum of a 15 Hz Ricker wavelet with a seeded delay and amplitude."""
    ow, dw = _band(c)
    r = np.random.default_rng(seed)
    f = ow + dw * np.arange(c["nw"])
    t = np.arange(512) * 0.004
    out = []
    for _ in range(nsrc):
        t0, amp = r.uniform(0.08, 0.15), r.uniform(0.8, 1.2)
        a = (np.pi * 15.0 * (t - t0)) ** 2
        out.append(amp * (np.exp(-2j * np.pi * np.outer(f, t)) @ ((1 - 2 * a) * np.exp(-a))))
    return torch.as_tensor(np.array(out).astype(np.complex64))


def _geometry(c, seed):
    """One surface source per shot at a seeded place between the nodes; receivers on
    every surface node (windows: on the node square around each shot's source)."""
    r = np.random.default_rng(seed + 7)
    nx, ny, ns = c["nx"], c["ny"], c["ns"] if c["op"] != "batch" else 1
    sx, sy, rx, ry, rid = [], [], [], [], []
    for s in range(ns):
        fx, fy = r.uniform(0.3, 0.7, 2)
        if c["op"] == "windows":
            fx = 0.3 if s == 0 else 0.68
        sx.append(fx * (nx - 1) * D)
        sy.append(fy * (ny - 1) * D)
        ix, iy = np.arange(nx), np.arange(ny)
        if c["op"] == "windows":
            hx, hy = (nx * (28 + s)) // 100, (ny * (40 - 3 * s)) // 100
            mx, my = int(sx[-1] / D), ny // 2
            ix, iy = ix[max(0, mx - hx):mx + hx + 1], iy[max(0, my - hy):my + hy + 1]
        gx, gy = np.meshgrid(D * ix, D * iy)
        rx.append(gx.ravel())
        ry.append(gy.ravel())
        rid.append(np.full(gx.size, s))
    f = np.float32
    rx = np.concatenate(rx).astype(f)
    return dict(sx=np.array(sx, f), sy=np.array(sy, f), sz=np.zeros(ns, f), s_ids=np.arange(ns, dtype=np.int32),
                rx=rx, ry=np.concatenate(ry).astype(f), rz=np.zeros(len(rx), f),
                r_ids=np.concatenate(rid).astype(np.int32))


def _randc(shape, seed):
    return torch.randn(shape, dtype=C64, device=_dev(), generator=_gen(seed, _dev()))


def _inputs(c, seed):
    """The arrays of a case, from the seed alone."""
    op, dev = c["op"], _dev()
    if op == "batch":
        # uneven shots: aperture and band of each between 45 % and 100 % of the largest
        fr = [1.0, 0.8, 0.56, 0.48]
        sub = []
        for i in range(c["ns"]):
            nx, ny = (max(48, int(c[k] * fr[i])) for k in ("nx", "ny"))
            d = dict(c, op="migrate", nx=nx, ny=ny, nw=max(8, int(c["nw"] * (1 - 0.1 * i))), ns=1,
                     padx=_smooth7(nx) - nx, pady=_smooth7(ny) - ny)
            sub.append((d, _inputs(d, seed * 10 + i)))
        return dict(sub=sub)
    NY, NX = c["ny"] + c["pady"], c["nx"] + c["padx"]
    s2 = _slow2(c, seed)
    i = dict(s2=s2)
    if op in ("step", "downward"):
        # these operators take the reference's per-frequency model
        i["model"] = s2[:, None].to(C64).expand(-1, c["nw"], -1, -1).contiguous()
        i["m"] = _randc((c["ns"], c["nw"], NY, NX), seed + 1)
        i["d"] = _randc((c["ns"], c["nw"], NY, NX), seed + 2)
        return i
    i["geom"] = _geometry(c, seed)
    i["wavelet"] = _ricker(c, c["ns"], seed).to(dev)
    ntr = len(i["geom"]["rx"])
    den = (1.0 + 0.1 * _velocity(c["nz"], c["ny"], c["nx"], seed + 3) / 1500.0).float()
    nwm = c["nw"] if c.get("perfreq") else 1
    pair = [s2[:, None].to(C64), den[:, None].to(C64)]
    if nwm > 1:  # mild dispersion and attenuation along the band
        k = torch.arange(nwm, device=dev)[None, :, None, None] / nwm
        pair = [pair[0] * (1 - 0.01 * k) * (1 + 0.01j), pair[1].expand(-1, nwm, -1, -1)]
    i["model"] = [m.to(C64).contiguous() for m in pair]
    i["data"] = _randc((ntr, c["nw"]), seed + 4)
    if op == "born":
        g = (c["nz"], nwm, c["ny"], c["nx"])
        i["dmodel"] = [(i["model"][0] * 0.1 * _randc(g, seed + 5).real).contiguous(),
                       (0.05 * _randc(g, seed + 6).real).to(C64).contiguous()]
    if op == "fwi":
        i["s"] = torch.sqrt(s2).contiguous()
    return i


# ---------------------------------------------------------------- states and passes
def _plan(c, i, cache_depths=None):
    """A plan with its references, model and traces bound, as a program on the plan
    interface holds it."""
    ow, dw = _band(c)
    p = Plan(nx=c["nx"], ny=c["ny"], nw=c["nw"], ns=c["ns"], nz=c["nz"], dx=D, dy=D, dz=D, ow=ow, dw=dw,
             padx=c["padx"], pady=c["pady"], nref=c["nref"], eps=c["eps"], taperx=c["taper"], tapery=c["taper"],
             step=c["step"])
    sref, labels = _refs(i["model"][0], c["nref"], c["padx"], c["pady"])
    sref = sref.to(C64).expand(-1, -1, c["nw"]).contiguous()
    p.set_refs(sref, labels, phase_cache=cache_depths is None)
    if cache_depths is not None:
        p.enable_phase_cache(depths=cache_depths)
    p.set_model(*i["model"])
    g = i["geom"]
    return dict(plan=p, src=p.traces(g["sx"], g["sy"], g["sz"], g["s_ids"]),
                rec=p.traces(g["rx"], g["ry"], g["rz"], g["r_ids"]), wavelet=i["wavelet"])


def _zeros(*shape, dtype=C64):
    return torch.zeros(shape, dtype=dtype, device=_dev())


def prepare(case, seed):
    c, i = case, _inputs(case, seed)
    op = c["op"]
    st = dict(c=c)
    if op in ("step", "downward"):
        kind = {"pspi": CudaWEM.PSPI, "nsps": CudaWEM.NSPS}[c["step"]] if op == "step" else CudaWEM.Downward
        st["op"] = kind(i["m"], i["d"], i["model"], _par(c))
        if op == "step":
            st["op"].set_depth(c["nz"] // 2)
        st.update(m=i["m"], d=i["d"], out=torch.empty_like(i["m"]), adj=torch.empty_like(i["m"]))
    elif op == "model":
        st.update(_plan(c, i))
        w = (c["nz"],) + st["plan"].wshape
        st.update(data=_zeros(*i["data"].shape), down=_zeros(*w), up=_zeros(*w))
    elif op == "migrate":
        st.update(_plan(c, i))
        st.update(data=i["data"], image=_zeros(c["nz"], c["ny"], c["nx"], dtype=torch.float32))
    elif op == "batch":
        st["inst"] = []
        for d, j in i["sub"]:
            e = _plan(d, j, cache_depths=1)  # one level of phase factors, as the batched job binds
            e.update(data=j["data"], image=_zeros(d["nz"], d["ny"], d["nx"], dtype=torch.float32))
            st["inst"].append(e)
        st["streams"] = [torch.cuda.Stream() for _ in range(4)]
    elif op in ("windows", "born"):
        par = _par(c)
        if c.get("rate"):
            par["compress_rate"] = c["rate"]
        st["model"] = i["model"]
        st["data"] = _zeros(*i["data"].shape)
        nb = (2, 2) if op == "windows" else (1, 1)
        st["prop"] = CudaWEM.Propagator(i["model"], st["data"], i["wavelet"], par, i["geom"], nb)
        if op == "born":
            # the background of the current model is there, as after the modelling
            st["prop"].forward(False, st["model"], st["data"])
            st["born"] = CudaWEM.ExtendedBorn(i["dmodel"], st["data"], st["model"], st["prop"])
            st.update(dmodel=i["dmodel"], res=i["data"], grad=[torch.empty_like(m) for m in i["dmodel"]])
    else:
        st.update(s=i["s"].requires_grad_(True), wavelet=i["wavelet"], geom=i["geom"], obs=i["data"],
                  par=_par(c, checkpoint=c.get("checkpoint")))
    return st


def run(st):
    op = st["c"]["op"]
    if op == "step" or op == "downward":
        st["op"].forward(False, st["m"], st["out"])
        st["op"].adjoint(False, st["adj"], st["d"])
        return st["out"], st["adj"]
    if op == "model":
        st["plan"].propagate(st["src"], st["rec"], st["wavelet"], st["data"], st["down"], st["up"])
        return st["data"], st["down"], st["up"]
    if op == "migrate":
        st["plan"].migrate(st["src"], st["rec"], st["wavelet"], st["data"], st["image"])
        return st["image"]
    if op == "batch":
        sweep(L.SWEEP_IMAGE, st["inst"], st["streams"])
        return [e["image"] for e in st["inst"]]
    if op == "windows":
        st["prop"].forward(False, st["model"], st["data"])
        return st["data"]
    if op == "born":
        st["born"].forward(False, st["dmodel"], st["data"])
        st["born"].adjoint(False, st["grad"], st["res"])
        return st["data"], st["grad"]
    J = FWIGradient.apply(st["s"], st["wavelet"], st["geom"], st["obs"], st["par"])
    return J.detach(), torch.autograd.grad(J, st["s"])[0]


# ---------------------------------------------------------------- what a pass needs
def work(case):
    """Bytes: inputs read once, outputs written once.  Flops: the 2D transforms of
    every depth step (nref + 1) and scattering (taylor + 2), 5 N log2 N each, and one
    complex multiplication per sample and term."""
    c, op = case, case["op"]
    if op == "batch":
        ws = []
        for f, i in zip([1.0, 0.8, 0.56, 0.48], range(c["ns"])):
            ws.append(work(dict(c, op="migrate", nx=max(48, int(c["nx"] * f)), ny=max(48, int(c["ny"] * f)),
                                nw=max(8, int(c["nw"] * (1 - 0.1 * i))), ns=1)))
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    NX, NY = c["nx"] + c["padx"], c["ny"] + c["pady"]
    shots = c["ns"] * (0.5 if op == "windows" else 1)  # each window covers about half of the model
    cells = NX * NY * c["nw"] * shots
    tr = 5 * math.log2(NX * NY) * cells
    stepf = (c["nref"] + 1) * tr + 6 * c["nref"] * cells
    scatf = 3 * tr + 12 * cells
    nz, wf = c["nz"], 8.0 * cells
    model = 8.0 * nz * c["ny"] * c["nx"] * (c["nw"] if c.get("perfreq") else 1)
    traces = 8.0 * c["nx"] * c["ny"] * c["nw"] * shots
    labels = nz * NX * NY * (c["nw"] if c.get("perfreq") or op in ("step", "downward") else 1)
    if op == "step":
        return {"bytes": 4 * wf + 2 * labels / nz, "flops": 2 * stepf}
    if op == "downward":
        return {"bytes": 4 * wf + 2 * labels, "flops": 2 * nz * stepf}
    if op == "model":
        return {"bytes": 2 * nz * wf + 2 * model + labels + traces, "flops": 2 * nz * stepf}
    if op == "windows":
        return {"bytes": 2 * model + labels + traces, "flops": 2 * nz * stepf}
    if op == "migrate":
        return {"bytes": 4.0 * nz * c["ny"] * c["nx"] + labels + traces, "flops": 2 * nz * stepf}
    if op == "born":
        store = wf * (16.5 / 32 if c.get("rate") else 1)
        # both background fields read by each operator; perturbation in, gradient out
        return {"bytes": 4 * nz * store + 6 * model + 2 * traces + 2 * labels, "flops": 4 * nz * (stepf + scatf)}
    # gradient: modelling down and up, the adjoint recursions, the derivatives
    return {"bytes": 4.0 * nz * c["ny"] * c["nx"] * 2 + traces, "flops": 4 * nz * stepf}


# ---------------------------------------------------------------- 64-bit results
def _refs(s2, nref, padx, pady):
    """References (squares of the slowness quantiles (2k+1)/(2 nref) of each
    (depth, frequency) row) [nz][nref][nw'] and nearest-reference labels
    [nz][nw'][NY][NX], edge-replicated into the pad."""
    nz, nw, ny, nx = s2.shape
    x = s2.reshape(nz * nw, ny * nx).to(C128)
    srt = torch.sort(torch.sqrt(x.real.clamp(min=0)), dim=1)[0]
    pos = (2 * torch.arange(nref, device=x.device, dtype=F64) + 1) / (2 * nref) * (ny * nx - 1)
    lo = pos.floor().long()
    hi = (lo + 1).clamp(max=ny * nx - 1)
    q = (srt[:, lo] * (1 - (pos - lo)) + srt[:, hi] * (pos - lo)) ** 2
    lab, best = None, None
    for r in range(nref):
        d = (x - q[:, r:r + 1]).abs()
        if r == 0:
            lab, best = torch.zeros_like(d, dtype=torch.uint8), d
        else:
            near = d < best
            lab[near] = r
            best = torch.minimum(best, d)
    lab = lab.reshape(nz, nw, ny, nx)
    iy = torch.arange(ny + pady, device=x.device).clamp(max=ny - 1)
    ix = torch.arange(nx + padx, device=x.device).clamp(max=nx - 1)
    return q.reshape(nz, nw, nref).permute(0, 2, 1), lab[:, :, iy][:, :, :, ix].contiguous()


class _Exact:
    """The depth-stepping operators in 64 bits on one grid."""

    def __init__(self, c, s2, den=None, ox=0.0, oy=0.0, f0=0):
        self.c, dev = c, s2.device
        self.nx, self.ny, self.nz, self.nw, self.ns = c["nx"], c["ny"], c["nz"], c["nw"], c["ns"]
        self.NX, self.NY = c["nx"] + c["padx"], c["ny"] + c["pady"]
        self.ox, self.oy = ox, oy
        ow, dw = c["band"] if "band" in c else _band(c)
        self.w = 2 * math.pi * (ow + dw * (f0 + torch.arange(self.nw, device=dev, dtype=F64)))
        kx, ky = (2 * math.pi * torch.fft.fftfreq(n, D, device=dev, dtype=F64) for n in (self.NX, self.NY))
        self.k2 = kx[None, :] ** 2 + ky[:, None] ** 2
        self.taper = self._tap(self.NY, dev)[:, None] * self._tap(self.NX, dev)[None, :]
        self.s2 = s2.to(C128)
        self.den = None if den is None else den.to(C128)
        self.sref, self.lab = _refs(s2, c["nref"], c["padx"], c["pady"])
        self.shape = (self.ns, self.nw, self.NY, self.NX)
        self.cache = {}

    def _tap(self, n, dev):
        t, i = self.c["taper"], torch.arange(n, device=dev, dtype=F64)
        w = torch.ones(n, device=dev, dtype=F64)
        if t:
            w = torch.where(i >= n - t, 0.5 * (1 + torch.cos(math.pi * (i - n + t) / t)), w)
            w = torch.where(i < t, 0.5 * (1 - torch.cos(math.pi * i / t)), w)
        return w

    def zero(self):
        return torch.zeros(self.shape, dtype=C128, device=self.w.device)

    def phase(self, sr, adjoint):
        """exp(-i kz dz) of the real references sr [nw]; the adjoint's is its conjugate
        (b <= 0 for these references, so no sign changes)."""
        a = (self.w ** 2 * sr)[:, None, None] - self.k2
        b = -(self.w ** 2 * self.c["eps"] * sr)[:, None, None]
        c = torch.sqrt(a * a + b * b)
        re = torch.sqrt((c + a).clamp(min=0) / 2)
        im = torch.sqrt((c - a).clamp(min=0) / 2)
        if self.c["eps"]:  # the smaller root from re im = |b| / 2, without the cancellation
            re, im = torch.where(a >= 0, re, b.abs() / 2 / im), torch.where(a >= 0, b.abs() / 2 / re, im)
        p = torch.exp(torch.complex(-im * D, -re * D))
        return p.conj() if adjoint else p

    def phases(self, iz, adjoint):
        sr = self.sref[iz].expand(-1, self.nw)
        return [self.phase(sr[r], adjoint) for r in range(self.c["nref"])]

    def fwd(self, iz, u, kind=None):
        lab = self.lab[iz][None]
        if (kind or self.c["step"]) == "pspi":
            U = torch.fft.fft2(u * self.taper)
            out = torch.zeros_like(u)
            for r, p in enumerate(self.phases(iz, False)):
                out += (lab == r) * torch.fft.ifft2(U * p)
            return out
        U = torch.zeros_like(u)
        for r, p in enumerate(self.phases(iz, False)):
            U += p * torch.fft.fft2((lab == r) * u)
        return torch.fft.ifft2(U)

    def adj(self, iz, u, kind=None, taper=True):
        lab = self.lab[iz][None]
        if (kind or self.c["step"]) == "pspi":
            U = torch.zeros_like(u)
            for r, p in enumerate(self.phases(iz, True)):
                U += p * torch.fft.fft2((lab == r) * u)
            return torch.fft.ifft2(U) * (self.taper if taper else 1.0)
        U = torch.fft.fft2(u)
        out = torch.zeros_like(u)
        for r, p in enumerate(self.phases(iz, True)):
            out += (lab == r) * torch.fft.ifft2(U * p)
        return out

    # -- acquisition: (cells, weights) of surface traces; all depths here are 0
    def traces(self, cx, cy, ids):
        f = np.float32
        ox, oy = f(self.ox), f(self.oy)
        ix = np.floor((cx - ox) / f(D)).astype(np.int64)
        iy = np.floor((cy - oy) / f(D)).astype(np.int64)
        lx = 1 - (cx.astype(np.float64) - (self.ox + ix * D)) / D
        ly = 1 - (cy.astype(np.float64) - (self.oy + iy * D)) / D
        ok = (ix >= 0) & (ix < self.NX - 1) & (iy >= 0) & (iy < self.NY - 1)
        t = lambda a: torch.as_tensor(a, device=self.w.device)  # noqa: E731
        cell = (np.asarray(ids).astype(np.int64) * self.NY + iy) * self.NX + ix
        w = [lx * ly, (1 - lx) * ly, lx * (1 - ly), (1 - lx) * (1 - ly)]
        off = [0, 1, self.NX, self.NX + 1]
        keep = t(np.nonzero(ok)[0])
        return keep, [t(cell[ok] + o) for o in off], [t(v[ok]) for v in w]

    def inject(self, tr, traces, u):
        keep, cells, ws = tr
        v = torch.zeros((self.ns * self.NY * self.NX, self.nw), dtype=C128, device=u.device)
        for q, w in zip(cells, ws):
            v.index_add_(0, q, w[:, None] * traces.to(C128)[keep])
        u += v.reshape(self.ns, self.NY, self.NX, self.nw).permute(0, 3, 1, 2)

    def record(self, tr, u, data):
        keep, cells, ws = tr
        v = u.permute(0, 2, 3, 1).reshape(-1, self.nw)
        data.index_add_(0, keep, sum(w[:, None] * v[q] for q, w in zip(cells, ws)))

    # -- model operators
    def pair(self, m, iz):
        return m[iz], m[min(iz + 1, self.nz - 1)]

    def refl(self, iz):
        (s0, s1), (r0, r1) = self.pair(self.s2, iz), self.pair(self.den, iz)
        a, b = r1 * torch.sqrt(s0), r0 * torch.sqrt(s1)
        return (a - b) / (a + b)

    def win(self, u):
        return u[:, :, :self.ny, :self.nx]

    def lin(self, iz):
        (s0, s1), (r0, r1) = self.pair(self.s2, iz), self.pair(self.den, iz)
        q0, q1 = torch.sqrt(s0), torch.sqrt(s1)
        inv2 = 1 / (r1 * q0 + r0 * q1) ** 2
        sc, ss, rr = torch.sqrt(q1 / q0), r0 * r1 * inv2, 2 * q0 * q1 * inv2
        return sc * ss, ss / sc, r0 * rr, r1 * rr

    def scatter(self, iz, u, adjoint):
        iy = torch.arange(self.NY, device=u.device).clamp(max=self.ny - 1)
        ix = torch.arange(self.NX, device=u.device).clamp(max=self.nx - 1)
        s = self.s2[iz][:, iy][:, :, ix]
        s = torch.complex(s.real, s.imag - 0.04 * s.real)
        w = self.w[:, None, None]
        out = torch.zeros_like(u)
        for n, cf in enumerate((1.0, 0.5)):
            W = -0.5j * w * D * cf * s ** (-0.5 - n)
            Q = (self.k2 / w ** 2) ** n
            if adjoint:
                out += torch.fft.ifft2(Q * torch.fft.fft2(W.conj() * u))
            else:
                out += W * torch.fft.ifft2(Q * torch.fft.fft2(u))
        return out

    # -- drivers
    def model(self, src, rec, wavelet, ntr, step=None):
        step = step or self.fwd
        data = torch.zeros((ntr, self.nw), dtype=C128, device=self.w.device)
        down, up, u = [], [None] * self.nz, self.zero()
        for iz in range(self.nz):
            if iz == 0:
                self.inject(src, wavelet, u)
                self.record(rec, u, data)
            down.append(u.clone())
            u = step(iz, u)
        u = self.zero()
        for iz in reversed(range(self.nz)):
            u = step(iz, u)
            self.win(u).add_(self.win(down[iz]) * self.refl(iz))
            if iz == 0:
                self.record(rec, u, data)
            up[iz] = u.clone()
        return data, down, up

    def migrate(self, src, rec, wavelet, data):
        S, R = self.zero(), self.zero()
        img = torch.zeros((self.nz, self.ny, self.nx), dtype=F64, device=S.device)
        for iz in range(self.nz):
            if iz == 0:
                self.inject(src, wavelet, S)
                self.inject(rec, data, R)
            img[iz] = (self.win(S).conj() * self.win(R)).real.sum(dim=(0, 1))
            S, R = self.fwd(iz, S), self.adj(iz, R)
        return img

    def _sum(self, g, like):
        return g.sum(0, keepdim=True) if like.shape[1] == 1 else g

    def born(self, rec, down, up, dm, ntr):
        ds, dr = (m.to(C128) for m in dm)
        data = torch.zeros((ntr, self.nw), dtype=C128, device=ds.device)
        u, store = self.zero(), []
        for iz in range(self.nz):  # down scattering (zero at the surface, so nothing is recorded)
            store.append(u.clone())
            sc = self.zero()
            self.win(sc).copy_(self.win(down[iz]) * ds[iz])
            u = self.fwd(iz, u + self.scatter(iz, sc, False))
        u = self.zero()
        for iz in reversed(range(self.nz)):  # up scattering, reflections
            if iz + 1 < self.nz:
                sc = self.zero()
                self.win(sc).copy_(self.win(up[iz + 1]) * ds[iz + 1])
                u = self.fwd(iz, u + self.scatter(iz, sc, False))
            self.win(u).add_(self.win(store[iz]) * self.refl(iz))
            (a, b, e, f), (d0, d1), (p0, p1) = self.lin(iz), self.pair(ds, iz), self.pair(dr, iz)
            if iz + 1 < self.nz:
                self.win(u).add_(self.win(down[iz]) * (a * d0 - b * d1 + e * p1 - f * p0))
            if iz == 0:
                self.record(rec, u, data)
        return data

    def born_adjoint(self, rec, down, up, data, like):
        gs, gr = (torch.zeros(like.shape, dtype=C128, device=like.device) for _ in range(2))
        ic = lambda bg, v: (self.win(bg).conj() * self.win(v)).sum(0)  # noqa: E731
        z, store = self.zero(), []
        for iz in range(self.nz):
            if iz > 0:
                sc = self.scatter(iz - 1, self.adj(iz - 1, z, taper=False), True)
                gs[iz] += self._sum(ic(up[iz], sc), like)
                z = self.adj(iz - 1, z)
            else:
                self.inject(rec, data, z)
            if iz + 1 < self.nz:
                g, (a, b, e, f) = ic(down[iz], z), self.lin(iz)
                gs[iz] += self._sum(a.conj() * g, like)
                gs[iz + 1] -= self._sum(b.conj() * g, like)
                gr[iz] -= self._sum(f.conj() * g, like)
                gr[iz + 1] += self._sum(e.conj() * g, like)
            store.append(z.clone())
        u = self.zero()
        for iz in reversed(range(self.nz)):
            sc = self.scatter(iz, self.adj(iz, u, taper=False), True)
            gs[iz] += self._sum(ic(down[iz], sc), like)
            u = self.adj(iz, u)
            self.win(u).add_(self.win(store[iz]) * self.refl(iz).conj())
        return [gs, gr]


class _ExactSmooth(_Exact):
    """The differentiable step (hat weights between the bracketing references, split
    step correction) and the adjoint-state gradient, in 64 bits."""

    def __init__(self, c, s):
        super().__init__(c, (s.double() ** 2)[:, None].to(C128), torch.ones_like(s)[:, None])
        s = s.double()
        lo, hi = s.amin(dim=(1, 2)), s.amax(dim=(1, 2))
        mid, half = 0.5 * (lo + hi), 0.5 * (hi - lo)
        half = torch.maximum(half, 0.5e-3 * mid)
        lin = torch.linspace(-1.0, 1.0, c["nref"], dtype=F64, device=s.device)
        self.refs = (mid[:, None] + half[:, None] * lin).float().double()  # 32-bit inputs of the step
        iy = torch.arange(self.NY, device=s.device).clamp(max=self.ny - 1)
        ix = torch.arange(self.NX, device=s.device).clamp(max=self.nx - 1)
        self.s, self.sp = s, s[:, iy][:, :, ix]

    def terms(self, iz, adjoint):
        sp, refs, n = self.sp[iz], self.refs[iz], self.c["nref"]
        j = (torch.searchsorted(refs, sp.contiguous(), right=True) - 1).clamp(0, n - 2)
        span = refs[j + 1] - refs[j]
        t = (sp - refs[j]) / span
        inside = (sp > refs[0]) & (sp < refs[-1])
        for r in range(n):
            w = torch.where(j == r, 1 - t, torch.where(j + 1 == r, t, 0.0))
            dw = torch.where(j == r, -1 / span, torch.where(j + 1 == r, 1 / span, 0.0))
            w = torch.where(inside, w, torch.where(sp <= refs[0], float(r == 0), float(r == n - 1)))
            dw = torch.where(inside, dw, 0.0)
            ss = torch.exp(-1j * self.w[:, None, None] * (sp - refs[r]) * D)
            yield self.phase((refs[r] ** 2).expand(self.nw), adjoint), ss, w, dw

    def smooth(self, iz, u, deriv=False):
        U, out = torch.fft.fft2(u * self.taper), torch.zeros_like(u)
        for p, ss, w, dw in self.terms(iz, False):
            k = (dw - 1j * self.w[:, None, None] * D * w) if deriv else w
            out += k * ss * torch.fft.ifft2(U * p)
        return out

    def smooth_adj(self, iz, u):
        U = torch.zeros_like(u)
        for p, ss, w, _ in self.terms(iz, True):
            U += p * torch.fft.fft2(w * ss.conj() * u)
        return torch.fft.ifft2(U) * self.taper

    def objective(self, src, rec, wavelet, obs):
        data, down, up = self.model(src, rec, wavelet, obs.shape[0], self.smooth)
        res = data - obs.to(C128)
        J = 0.5 * (res.abs() ** 2).sum()
        cor = lambda a, b: (a.conj() * b).real.sum(dim=(0, 1))  # noqa: E731
        gp = torch.zeros((self.nz, self.NY, self.NX), dtype=F64, device=obs.device)
        g = torch.zeros_like(self.s)
        mu, mus = self.zero(), []
        for iz in range(self.nz):
            mu = self.smooth_adj(iz - 1, mu) if iz else mu
            if iz == 0:
                self.inject(rec, res, mu)
            mus.append(mu.clone())
            if iz + 1 < self.nz:
                gp[iz] += cor(mu, self.smooth(iz, up[iz + 1], True))
                k, s0, s1 = cor(self.win(mu), self.win(down[iz])), self.s[iz], self.s[iz + 1]
                g[iz] += k * 2 * s1 / (s0 + s1) ** 2
                g[iz + 1] -= k * 2 * s0 / (s0 + s1) ** 2
        nu = self.zero()
        for iz in reversed(range(self.nz)):
            if iz + 1 < self.nz:
                gp[iz] += cor(nu, self.smooth(iz, down[iz], True))
            nu = self.smooth_adj(iz, nu)
            self.win(nu).add_(self.win(mus[iz]) * self.refl(iz).conj())
        g += gp[:, :self.ny, :self.nx]  # the pad's cells repeat the edge's slowness
        g[:, :, -1] += gp[:, :self.ny, self.nx:].sum(2)
        g[:, -1, :] += gp[:, self.ny:, :self.nx].sum(1)
        g[:, -1, -1] += gp[:, self.ny:, self.nx:].sum((1, 2))
        return J, g


def _exact_shot(c, i):
    e = _Exact(c, i["model"][0], i["model"][1])
    g = i["geom"]
    return e, e.traces(g["sx"], g["sy"], g["s_ids"]), e.traces(g["rx"], g["ry"], g["r_ids"]), len(g["rx"])


def _exact_windows(c, i):
    """Every (shot, band) pair modelled on the box around its source and receivers."""
    g = i["geom"]
    out = torch.zeros((len(g["rx"]), c["nw"]), dtype=C128, device=i["s2"].device)
    ow, dw = _band(c)
    half = c["nw"] - c["nw"] // 2
    for s in range(2):
        rows = np.nonzero(g["r_ids"] == s)[0]
        box = []
        for a, n in (("x", c["nx"]), ("y", c["ny"])):
            p = np.concatenate([g["s" + a][s:s + 1], g["r" + a][rows]]).astype(np.float64)
            lo, hi = max(0, math.floor(p.min() / D)), min(n - 1, math.ceil(p.max() / D))
            box.append((lo, hi) if hi > lo else (0, n - 1))
        (x0, x1), (y0, y1) = box
        for f0, nf in ((0, half), (half, c["nw"] - half)):
            nx, ny = x1 - x0 + 1, y1 - y0 + 1
            d = dict(c, nx=nx, ny=ny, nw=nf, ns=1, padx=_smooth7(nx + c["padx"]) - nx,
                     pady=_smooth7(ny + c["pady"]) - ny, band=(ow, dw))
            m = [t[:, :, y0:y1 + 1, x0:x1 + 1].contiguous() for t in i["model"]]
            e = _Exact(d, m[0], m[1], x0 * D, y0 * D, f0)
            src = e.traces(g["sx"][s:s + 1], g["sy"][s:s + 1], [0])
            rec = e.traces(g["rx"][rows], g["ry"][rows], np.zeros(len(rows)))
            data = e.model(src, rec, i["wavelet"][s:s + 1, f0:f0 + nf], len(rows))[0]
            out[torch.as_tensor(rows, device=out.device), f0:f0 + nf] += data
    return out


def exact(case, seed):
    c, i, op = case, _inputs(case, seed), case["op"]
    if op == "batch":
        out = []
        for d, j in i["sub"]:
            e, src, rec, _ = _exact_shot(d, j)
            out.append(e.migrate(src, rec, j["wavelet"], j["data"]))
        return out
    if op in ("step", "downward"):
        e = _Exact(c, i["model"])
        m, d = i["m"].to(C128), i["d"].to(C128)
        if op == "step":
            iz = c["nz"] // 2
            # the single-step adjoint leaves the taper out
            return e.fwd(iz, m), e.adj(iz, d, taper=False)
        for iz in range(c["nz"]):
            m = e.fwd(iz, m)
        for iz in reversed(range(c["nz"])):
            d = e.adj(iz, d)
        return m, d
    if op == "windows":
        return _exact_windows(c, i)
    if op == "fwi":
        e, g = _ExactSmooth(c, i["s"]), i["geom"]
        return e.objective(e.traces(g["sx"], g["sy"], g["s_ids"]), e.traces(g["rx"], g["ry"], g["r_ids"]),
                           i["wavelet"], i["data"])
    e, src, rec, ntr = _exact_shot(c, i)
    if op == "model":
        data, down, up = e.model(src, rec, i["wavelet"], ntr)
        return data, torch.stack(down), torch.stack(up)
    if op == "migrate":
        return e.migrate(src, rec, i["wavelet"], i["data"])
    _, down, up = e.model(src, rec, i["wavelet"], ntr)
    return (e.born(rec, down, up, i["dmodel"], ntr),
            e.born_adjoint(rec, down, up, i["data"], i["dmodel"][0]))

"""Performance cases of the viscoelastic time step: what a user has the
framework do, through its public entry points.

A case is a dict of plain values; its "call" names the entry point:

  step      StepPlan.step: a chunk of a time loop on device-resident fields,
            sources and receivers included (a whole solve is many of these)
  leapfrog  api.leapfrog_step_: one blocking step of an isotropic medium,
            the reference's own entry point and the smallest call there is
  solve     StepPlan.forward_host: one whole solve from host buffers, medium
            and wavelet up, traces down
  gather    batch.ShotBatch: a gather of shots of different grids and step
            counts, from rest to their ends
  gradient  gradient.shot_misfit and its backward (FP32), or
            gradient.misfit_gradient (FP64): the misfit of one shot and its
            gradient with respect to every medium plane

prepare() makes the inputs on the GPU from the seed, run() is one pass, and
exact() is the same computation in plain torch at 64 bits (the gradient by
torch.autograd through it).
"""
import math

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from viscoelasticinversion_b200 import CPMLSpec, StepPlan, api, make_config, media
from viscoelasticinversion_b200.batch import ShotBatch
from viscoelasticinversion_b200.gradient import misfit_gradient, shot_misfit

H = 4  # half-length of the staggered stencil; cells nearer than this to an edge are never updated
DX, DT, F0, VMAX = 5.0, 0.4e-3, 12.0, 5800.0  # the layered workloads' spacing, step, source frequency
PLANES = {"iso": ("rho", "c13", "c55"), "vti": ("rho", "c11", "c13", "c33", "c55"),
          "tti": ("rho", "c11", "c13", "c15", "c33", "c35", "c55")}
SMALL_GRIDS = ((256, 256), (384, 256), (512, 256))  # shots that do not fill the GPU by themselves


def listed():
    return [
        # one step of a small model, waited for: latency, launches and the host path are everything
        {"name": "leapfrog iso 256x256", "call": "leapfrog", "kind": "iso", "nx": 256, "nz": 256, "prec": "f32",
         "nsls": 3, "pml": 20, "fs": True},
        # the reference's CPU-runnable forward model: 256 x 256 in FP64
        {"name": "step iso 256x256 f64", "call": "step", "kind": "iso", "nx": 256, "nz": 256, "prec": "f64", "nsls": 3,
         "pml": 20, "fs": True, "nsteps": 200},
        # the single-shot workload the framework quotes its rate on
        {"name": "step vti 2048x1024", "call": "step", "kind": "vti", "nx": 2048, "nz": 1024, "prec": "f32", "nsls": 3,
         "pml": 40, "fs": True, "nsteps": 100},
        # a tilted medium, ordinary size
        {"name": "step tti 1024x512", "call": "step", "kind": "tti", "nx": 1024, "nz": 512, "prec": "f32", "nsls": 3,
         "pml": 40, "fs": True, "nsteps": 200},
        # the largest model that requests bring: wider than every cache
        {"name": "step tti 4096x2048", "call": "step", "kind": "tti", "nx": 4096, "nz": 2048, "prec": "f32", "nsls": 3,
         "pml": 40, "fs": True, "nsteps": 30},
        # a model cut to its survey's extent: rows that are no multiple of a vector
        {"name": "step vti 1403x597", "call": "step", "kind": "vti", "nx": 1403, "nz": 597, "prec": "f32", "nsls": 3,
         "pml": 30, "fs": True, "nsteps": 60},
        # the compensated stresses of long runs, no free surface, two mechanisms
        {"name": "step iso 1536x768 f32c", "call": "step", "kind": "iso", "nx": 1536, "nz": 768, "prec": "f32c",
         "nsls": 2, "pml": 30, "fs": False, "nsteps": 100},
        # one whole solve, host to host
        {"name": "solve vti 512x512", "call": "solve", "kind": "vti", "nx": 512, "nz": 512, "prec": "f32", "nsls": 3,
         "pml": 40, "fs": True, "nsteps": 500},
        # a gather of small shots, each too small to fill the GPU
        {"name": "gather tti 12 shots", "call": "gather", "kind": "tti", "nx": 512, "nz": 256, "prec": "f32", "nsls": 3,
         "pml": 20, "fs": True, "shots": 12, "nsteps": 240},
        # one shot of an inversion: misfit and gradient, the forward states kept
        {"name": "gradient vti 1024x512", "call": "gradient", "kind": "vti", "nx": 1024, "nz": 512, "prec": "f32",
         "nsls": 3, "pml": 40, "fs": True, "nsteps": 160, "every": 0},
        # the same for a tilted medium, from checkpoints as the server runs it
        {"name": "gradient tti 512x384", "call": "gradient", "kind": "tti", "nx": 512, "nz": 384, "prec": "f32",
         "nsls": 3, "pml": 30, "fs": True, "nsteps": 144, "every": 12},
        # a checking run of the gradient: FP64 on an odd grid
        {"name": "gradient iso 301x203 f64", "call": "gradient", "kind": "iso", "nx": 301, "nz": 203, "prec": "f64",
         "nsls": 3, "pml": 20, "fs": True, "nsteps": 120, "every": 0},
    ]


def draw(rng):
    """One more case: any of the calls, sizes spread over the logarithm of
    their range, half of them multiples of 4 (what vectors like) and the
    others as they fall, and a step count that bounds the work."""
    call = rng.choices(("leapfrog", "step", "solve", "gather", "gradient"), (1, 6, 1, 1, 3))[0]

    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n if even else n | rng.randrange(2)

    even = rng.random() < 0.5 or call == "gather"
    top = {"leapfrog": (700, 500), "step": (4096, 2048), "solve": (1100, 700), "gather": (512, 256),
           "gradient": (1100, 600)}[call]
    nx, nz = size(160, top[0]), size(128, top[1])
    if even:
        nx -= nx % 4
    case = {"call": call, "kind": "iso" if call == "leapfrog" else rng.choice(("iso", "vti", "tti")), "nx": nx,
            "nz": nz, "prec": rng.choice(("f32", "f32", "f32", "f64")), "nsls": rng.choice((1, 2, 3, 3, 3)),
            "pml": rng.randrange(12, 41), "fs": rng.random() < 0.75}
    if call == "step" and even and rng.random() < 0.15:
        case["prec"] = "f32c"
    if call == "leapfrog":
        return case
    steps = {"step": 1.6e8, "solve": 0.8e8, "gather": 0, "gradient": 0.4e8}[call]
    case["nsteps"] = max(20, min(240, int(steps / (nx * nz)))) + rng.randrange(8)
    if call == "gather":
        case.update(shots=rng.randrange(4, 13), prec="f32", nsteps=rng.randrange(100, 220))
    if call == "gradient":
        case["every"] = rng.choice((0, 0, int(math.ceil(math.sqrt(case["nsteps"])))))
    return case


# ------------------------------------------------------------------ inputs


def _noise(g, nz, nx, cells, dev):
    """Smooth unit-variance noise of a correlation length of about `cells`."""
    a = torch.randn(1, 1, nz // cells + 3, nx // cells + 3, generator=g, device=dev, dtype=torch.float64)
    f = F.interpolate(a, size=(nz, nx), mode="bicubic", align_corners=False)[0, 0]
    return f / f.std()


def _uniform(g, n, lo, hi, dev):
    return lo + (hi - lo) * torch.rand(n, generator=g, device=dev, dtype=torch.float64)


def _qfit(nsls):
    return media.q_fit(2.0, 30.0, nsls)


def _medium(case, g, nx, nz, dev, smooth=1.0):
    """Eight layers with 3 % smooth perturbations (FP64 planes [nz, nx]);
    smooth < 1 scales the perturbations down (a starting model)."""
    depth = torch.arange(nz, device=dev, dtype=torch.float64)
    layer = torch.searchsorted(torch.sort(_uniform(g, 7, 0.05 * nz, 0.95 * nz, dev)).values, depth)
    vp = torch.sort(_uniform(g, 8, 1800.0, 4500.0, dev)).values[layer][:, None]
    eps = _uniform(g, 8, 0.0, 0.25, dev)[layer][:, None]
    dlt = _uniform(g, 8, -0.05, 0.15, dev)[layer][:, None]
    q = _uniform(g, 8, 30.0, 200.0, dev)[layer][:, None].expand(nz, nx)
    vp = vp * (1.0 + 0.03 * smooth * _noise(g, nz, nx, 10, dev).clamp(-3, 3))
    rho = 310.0 * vp**0.25 * (1.0 + 0.03 * smooth * _noise(g, nz, nx, 10, dev).clamp(-3, 3))
    th = _noise(g, nz, nx, 40, dev).clamp(-2, 2) * math.radians(15.0)
    c33, c55 = rho * vp**2, rho * (vp / 1.8) ** 2
    if case["kind"] == "iso":
        med = {"rho": rho, "c13": c33 - 2 * c55, "c55": c55}
    else:
        c11 = c33 * (1 + 2 * eps)
        c13 = torch.sqrt((c33 - c55) * (c33 * (1 + 2 * dlt) - c55)) - c55
        med = {"rho": rho, "c11": c11, "c13": c13, "c33": c33, "c55": c55}
        if case["kind"] == "tti":
            c, s = torch.cos(th), torch.sin(th)
            c2, s2, cs, a = c * c, s * s, c * s, c13 + 2 * c55
            med = {"rho": rho, "c11": c2 * c2 * c11 + 2 * c2 * s2 * a + s2 * s2 * c33,
                   "c13": c2 * s2 * (c11 + c33 - 4 * c55) + (c2 * c2 + s2 * s2) * c13,
                   "c15": -cs * (c2 * c11 - s2 * c33 - (c2 - s2) * a),
                   "c33": s2 * s2 * c11 + 2 * c2 * s2 * a + c2 * c2 * c33,
                   "c35": -cs * (s2 * c11 - c2 * c33 + (c2 - s2) * a),
                   "c55": c2 * s2 * (c11 + c33 - 2 * c13) + (c2 - s2) ** 2 * c55}
    if case["nsls"]:
        qf = _qfit(case["nsls"])
        med["tau"] = len(qf.taus) / (qf.Kbar * q)
    return {k: v.contiguous() for k, v in med.items()}


def _state(case, g, nx, nz, dev):
    """The fields in the middle of a solve: smooth noise of seismic size in
    the updated cells, zero around them, stress images above a surface."""
    n = case["nsls"]

    def planes(k, scale):
        out = torch.zeros(k, nz, nx, device=dev, dtype=torch.float64)
        for p in out:
            p[H:-H, H:-H] = scale * _noise(g, nz, nx, 8, dev)[H:-H, H:-H]
        return out

    v, s, m = planes(2, 1e-4), planes(3, 600.0), planes(3 * max(n, 1), 2e-7)
    if case["fs"]:
        s[1, H] = 0
        m[n:2 * n, H] = 0
        s[1, :H] = -s[1, H + 1:2 * H + 1].flip(0)
        s[2, :H] = -s[2, H:2 * H].flip(0)
    return {"v": v, "s": s, "m": m.view(3, max(n, 1), nz, nx)}


def _spread(nx, n, row):
    return [(int(i), row) for i in sorted({int(round(x)) for x in np.linspace(H + 8, nx - H - 9, n)})]


def _dtype(case):
    return torch.float64 if case["prec"] == "f64" else torch.float32


def _problem(case, seed):
    """Everything a case starts from, in its own precision, on the GPU."""
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 7919 + 17)
    dt = _dtype(case)
    to = lambda d: {k: t.to(dt).contiguous() for k, t in d.items()}  # noqa: E731
    nx, nz = case["nx"], case["nz"]
    if case["call"] == "gather":
        shots = []
        for q in range(case["shots"]):
            w, h = SMALL_GRIDS[q % 3]
            w, h = w * nx // 512 // 4 * 4, h * nz // 256
            nt = case["nsteps"] - q * case["nsteps"] // (2 * case["shots"])
            shots.append(dict(nx=w, nz=h, nt=nt, medium=to(_medium(case, g, w, h, dev)), sources=[(w // 2, H + 4, 0, 1e6)],
                              receivers=_spread(w, 64, H + 2)))
        return shots
    p = {"nx": nx, "nz": nz, "nt": case.get("nsteps", 1)}
    p["medium"] = to(_medium(case, g, nx, nz, dev))
    p["sources"] = [(nx // 2, H + 4, 0, 1e6)] if case["call"] != "leapfrog" else []
    p["receivers"] = _spread(nx, 256 if nx > 512 else 100, H + 2) if case["call"] != "leapfrog" else []
    if case["call"] in ("step", "leapfrog"):
        p["state"] = to(_state(case, g, nx, nz, dev))
    if case["call"] == "gradient":  # observed traces: a band-limited record of the size a solve gives
        t = _noise(g, len(p["receivers"]), p["nt"] + 64, 24, dev)[:, 32:32 + p["nt"]]
        u = _noise(g, len(p["receivers"]), p["nt"] + 64, 24, dev)[:, 32:32 + p["nt"]]
        p["obs"] = (1e-6 * torch.stack((t, u))).to(dt).contiguous()
    return p


def _wavelet(nt):
    """Ricker samples [1, nt] whose peak lies within the chunk."""
    x = math.pi * F0 * (np.arange(nt) * DT - min(1.2 / F0, 0.5 * nt * DT))
    return ((1.0 - 2.0 * x * x) * np.exp(-x * x))[None, :]


def _cpml(case):
    return CPMLSpec(thickness=case["pml"], alpha_max=math.pi * F0, top=not case["fs"], vmax=VMAX)


def _taus(case):
    return _qfit(case["nsls"]).taus if case["nsls"] else np.zeros(0)


def prepare(case, seed):
    call, p = case["call"], _problem(case, seed)
    if call == "gather":
        works = [media.Workload(
            name="shot%d" % q, nx=s["nx"], nz=s["nz"], dx=DX, dz=DX, dt=DT, nt=s["nt"], kind=case["kind"],
            medium={k: t.double().cpu().numpy() for k, t in s["medium"].items()}, taus=_taus(case),
            free_surface=int(case["fs"]), pml=case["pml"], pml_vmax=VMAX, pml_alpha_max=math.pi * F0,
            sources=s["sources"], wavelets=_wavelet(s["nt"]), receivers=s["receivers"], vmax=VMAX)
            for q, s in enumerate(p)]
        return {"call": call, "batch": ShotBatch(works, case["prec"])}
    if call == "leapfrog":
        med, st = p["medium"], p["state"]
        return {"call": call, "fields": api.Fields(st["s"], st["m"], st["v"]),
                "parameters": api.Parameters(med["c13"], med["c55"], med.get("tau"), _taus(case), ρs=med["rho"], dx=DX,
                                             cpml=_cpml(case), free_surface=case["fs"])}
    plan = StepPlan(make_config(p["nx"], p["nz"], DX, DX, DT, case["kind"], case["prec"], _taus(case), case["fs"],
                                _cpml(case)))
    wav = torch.as_tensor(_wavelet(p["nt"]), dtype=plan.dtype)
    p.update(call=call, plan=plan, every=case.get("every", 0))
    if call == "solve":
        p["medium"] = {k: t.cpu().pin_memory() for k, t in p["medium"].items()}
        p["wavelets"] = wav.pin_memory()
        p["traces"] = torch.empty(2, len(p["receivers"]), p["nt"], dtype=plan.dtype).pin_memory()
    else:
        p["wavelets"] = wav.to(plan.device)
        p["traces"] = torch.zeros(2, len(p["receivers"]), p["nt"], dtype=plan.dtype, device=plan.device)
    return p


def run(state):
    call, p = state["call"], state
    if call == "leapfrog":
        f = p["fields"]
        api.leapfrog_step_(f, p["parameters"], DT)
        return {"v": f.v, "s": f.s, "m": f.M}
    if call == "gather":
        b = p["batch"]
        b.reset()
        b.run()
        return [{"traces": t, **s} for t, s in zip(b.traces, b.states)]
    if call == "step":
        p["plan"].step(p["medium"], p["state"], nsteps=p["nt"], sources=p["sources"], wavelets=p["wavelets"],
                       receivers=p["receivers"], traces=p["traces"])
        return {"traces": p["traces"], **p["state"]}
    if call == "solve":
        return p["plan"].forward_host(p["medium"], p["sources"], p["wavelets"], p["receivers"], p["nt"],
                                      traces_out=p["traces"])
    if p["plan"].dtype == torch.float64:
        misfit, grad = misfit_gradient(p["plan"], p["medium"], p["sources"], p["wavelets"], p["receivers"], p["obs"],
                                       checkpoint_every=p["every"])
        return {"misfit": misfit, "gradient": grad}
    planes = {k: t.detach().requires_grad_() for k, t in p["medium"].items()}
    misfit = shot_misfit(p["plan"], planes, p["sources"], p["wavelets"], p["receivers"], p["obs"],
                         checkpoint_every=p["every"])
    grads = torch.autograd.grad(misfit, list(planes.values()))
    return {"misfit": misfit.item(), **dict(zip(planes, grads))}


def work(case):
    """Counted per time step, the unit of the framework's roofline: each state
    plane (v, sigma, memory variables, CPML strips) read and written once and
    each medium plane read once; an adjoint step also reads the forward state,
    and reads and writes its own state and the FP64 gradient planes.  A grid
    that stays in the caches over the steps of a call can beat it."""
    size = 8 if case["prec"] == "f64" else 4
    n = case["nsls"]
    medium = len(PLANES[case["kind"]]) + (1 if n else 0)
    state = 5 + 3 * n
    nx, nz, nt = case["nx"], case["nz"], case.get("nsteps", 1)
    cells = nx * nz
    if case["call"] == "gather":  # grids of 256 .. 512 by 256, half to all of the step count
        cells, nt = cells * 0.75, nt * 0.75 * case["shots"]
    strips = 8 * case["pml"] * (2 * nz + nx * (1 if case["fs"] else 2))
    step = size * (cells * (2 * state + medium) + strips) + (6 * cells if case["prec"] == "f32c" else 0)
    flops = cells * (112 + 21 * n + (40 if case["kind"] == "tti" else 0))
    if case["call"] == "gradient":
        step += size * (cells * (3 * state + medium) + 1.5 * strips) + 16 * cells * medium
        flops *= 3
    return {"bytes": nt * step, "flops": nt * flops}


# ------------------------------------------------- the same in plain torch


def _d(u, axis, sign, n):
    """Staggered 8th-order derivative of the plane u over the updated cells:
    at the half node above (sign > 0) or below along the axis."""
    w = (1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168)
    nz, nx = u.shape
    out = 0
    for k in range(4):
        a, b = (k + 1, -k) if sign > 0 else (k, -k - 1)
        if axis == 1:
            t = u[H:nz - H, H + a:nx - H + a] - u[H:nz - H, H + b:nx - H + b]
        else:
            t = u[H + a:nz - H + a, H:nx - H] - u[H + b:nz - H + b, H:nx - H]
        out = out + (w[k] / DX) * t
    return out


def _profile(case, n, half, lo, hi, dev):
    """1/kappa, a, b of the CPML recursion at the updated nodes of one axis."""
    x = torch.arange(n, device=dev, dtype=torch.float64) + (0.5 if half else 0.0)
    lp = case["pml"]
    p = torch.zeros_like(x)
    if lo:
        p = torch.maximum(p, (lp - 0.5 - x) / lp)
    if hi:
        p = torch.maximum(p, (x - (n - lp - 0.5)) / lp)
    d0 = -3.0 * VMAX * math.log(1e-5) / (2.0 * lp * DX)
    d = torch.where(p > 0, d0 * p * p, 0.0)
    al = torch.where(p > 0, math.pi * F0 * (1.0 - p), 0.0)
    b = torch.where(p > 0, torch.exp(-(d + al) * DT), 0.0)
    a = torch.where(p > 0, d / (d + al).clamp_min(1e-300) * (b - 1.0), 0.0)
    return a[H:n - H], b[H:n - H]  # kappa is 1 throughout


class _Exact:
    """The leapfrog step on the updated cells in 64 bits, out of place."""

    def __init__(self, case, nx, nz, medium, taus, sources, receivers, wavelet):
        self.case, self.nx, self.nz = case, nx, nz
        self.taus = [float(t) for t in taus]
        dev = medium["rho"].device
        fs = case["fs"]
        self.fs = fs
        x = [_profile(case, nx, h, True, True, dev) for h in (0, 1)]
        z = [[t[:, None] for t in _profile(case, nz, h, not fs, True, dev)] for h in (0, 1)]
        # (a, b) of the eight derivatives in the order of psi
        self.ab = [x[1], z[0], x[0], z[1], x[0], z[0], z[1], x[1]]
        self.sources, self.wavelet = sources, wavelet
        self.rj = torch.tensor([j - H for _, j in receivers], device=dev)
        self.ri = torch.tensor([i - H for i, _ in receivers], device=dev)
        self.set_medium(medium)

    def set_medium(self, m):
        nx, nz, kind = self.nx, self.nz, self.case["kind"]
        inner = lambda u: u[H:nz - H, H:nx - H]  # noqa: E731
        half = lambda u: 0.25 * (u[H:nz - H, H:nx - H] + u[H:nz - H, H + 1:nx - H + 1] +  # noqa: E731
                                 u[H + 1:nz - H + 1, H:nx - H] + u[H + 1:nz - H + 1, H + 1:nx - H + 1])
        r = m["rho"]
        self.bx = 2.0 / (inner(r) + r[H:nz - H, H + 1:nx - H + 1])
        self.bz = 2.0 / (inner(r) + r[H + 1:nz - H + 1, H:nx - H])
        self.c13 = inner(m["c13"])
        self.c11 = inner(m["c11"]) if kind != "iso" else self.c13 + 2.0 * inner(m["c55"])
        self.c33 = inner(m["c33"]) if kind != "iso" else self.c11
        self.c55h = half(m["c55"])
        if kind == "tti":
            self.c15, self.c35, self.c15h, self.c35h = inner(m["c15"]), inner(m["c35"]), half(m["c15"]), half(m["c35"])
        self.tau = inner(m["tau"]) if self.taus else None

    def start(self, state=None):
        """[vx, vz, sxx, szz, sxz, M..., psi...] on the updated cells."""
        n, shape = 3 * len(self.taus), (self.nz - 2 * H, self.nx - 2 * H)
        zero = torch.zeros(shape, device=self.bx.device, dtype=torch.float64)
        if state is None:
            return [zero] * (5 + n + 8)
        inner = [p[H:-H, H:-H].double() for q in ("v", "s", "m") for p in state[q].reshape(-1, self.nz, self.nx)]
        return inner[:5 + n] + [zero] * 8

    def _full(self, u, image=None):
        """The plane with its images above the surface, zero around it."""
        if self.fs and image is not None:
            top = -(u[1:H + 1] if image == "szz" else u[:H]).flip(0)
            return F.pad(torch.cat((top, u)), (H, H, 0, H))
        return F.pad(u, (H, H, H, H))

    def step(self, st, it):
        vx, vz, sxx, szz, sxz = st[:5]
        n = len(self.taus)
        m, psi = list(st[5:5 + 3 * n]), list(st[5 + 3 * n:])

        def cpml(q, d):
            a, b = self.ab[q]
            psi[q] = b * psi[q] + a * d
            return d + psi[q]

        fxx, fzz, fxz = self._full(sxx), self._full(szz, "szz"), self._full(sxz, "sxz")
        vx = vx + DT * self.bx * (cpml(0, _d(fxx, 1, 1, 0)) + cpml(1, _d(fxz, 0, -1, 0)))
        vz = vz + DT * self.bz * (cpml(2, _d(fxz, 1, -1, 0)) + cpml(3, _d(fzz, 0, 1, 0)))
        traces = torch.stack((vx[self.rj, self.ri], vz[self.rj, self.ri])) if len(self.ri) else None
        fvx, fvz = self._full(vx), self._full(vz)
        rxx, rzz = cpml(4, _d(fvx, 1, -1, 0)), cpml(5, _d(fvz, 0, -1, 0))
        rxz = cpml(6, _d(fvx, 0, 1, 0)) + cpml(7, _d(fvz, 1, 1, 0))
        e = [rxx, rzz, rxz]
        if n:
            e = [(1.0 + self.tau) * r + self.tau * sum(m[q * n:(q + 1) * n]) for q, r in enumerate(e)]
        exx, ezz, exz = e
        tti = self.case["kind"] == "tti"
        ebxz = 0.0
        if tti:
            p = F.pad(exz, (1, 0, 1, 0))
            ebxz = 0.25 * (p[1:, 1:] + p[1:, :-1] + p[:-1, 1:] + p[:-1, :-1])
        if self.fs:  # the vertical rate on the surface follows from szz = 0
            num = self.c13[:1] * exx[:1] + (self.c35[:1] * ebxz[:1] if tti else 0.0)
            ezz = torch.cat((-num / self.c33[:1], ezz[1:]))
        dxx, dzz, dxz = self.c11 * exx + self.c13 * ezz, self.c13 * exx + self.c33 * ezz, self.c55h * exz
        if tti:
            px, pz = F.pad(exx, (0, 1, 0, 1)), F.pad(ezz, (0, 1, 0, 1))
            mean = lambda u: 0.25 * (u[:-1, :-1] + u[:-1, 1:] + u[1:, :-1] + u[1:, 1:])  # noqa: E731
            dxx, dzz = dxx + self.c15 * ebxz, dzz + self.c35 * ebxz
            dxz = dxz + self.c15h * mean(px) + self.c35h * mean(pz)
        sxx, szz, sxz = sxx + DT * dxx, szz + DT * dzz, sxz + DT * dxz
        for q, r in enumerate((rxx, rzz, rxz)):
            for k, t in enumerate(self.taus):
                new = m[q * n + k] + DT * (-r / (n * t) - m[q * n + k] / t)
                if self.fs and q == 1:
                    new = torch.cat((torch.zeros_like(new[:1]), new[1:]))
                m[q * n + k] = new
        for (i, j, _, amp), w in zip(self.sources, self.wavelet):
            add = torch.zeros_like(sxx)
            add[j - H, i - H] = DT * amp * float(w[it])
            sxx, szz = sxx + add, szz + add
        if self.fs:
            szz = torch.cat((torch.zeros_like(szz[:1]), szz[1:]))
        return [vx, vz, sxx, szz, sxz] + m + psi, traces

    def run(self, st, nt):
        rows = []
        for it in range(nt):
            st, t = self.step(st, it)
            rows.append(t)
        return st, torch.stack(rows, -1) if rows[0] is not None else None

    def fields(self, st):
        """v, s, m as the framework lays them out."""
        n = len(self.taus)
        v = torch.stack([self._full(u) for u in st[:2]])
        s = torch.stack([self._full(st[2]), self._full(st[3], "szz"), self._full(st[4], "sxz")])
        m = torch.stack([self._full(u) for u in st[5:5 + 3 * n]]).view(3, n, self.nz, self.nx) if n else \
            torch.zeros(3, 1, self.nz, self.nx, device=v.device, dtype=v.dtype)
        return {"v": v, "s": s, "m": m}


def _exact_gradient(case, p, wavelet):
    """Misfit and gradients by torch.autograd, the steps recomputed in runs
    of ten on the way back so the graph fits the card."""
    names = list(p["medium"])
    leaves = [p["medium"][k].double().requires_grad_() for k in names]
    sim = _Exact(case, p["nx"], p["nz"], p["medium"], _taus(case), p["sources"], p["receivers"], wavelet)
    obs = p["obs"].double()
    sim.set_medium({k: t.detach() for k, t in zip(names, leaves)})
    st = sim.start()

    def chunk(it0, it1, *args):
        sim.set_medium(dict(zip(names, args[:len(names)])))
        cur, part = list(args[len(names):]), 0.0
        for it in range(it0, it1):
            cur, t = sim.step(cur, it)
            part = part + 0.5 * ((t - obs[:, :, it]) ** 2).sum()
        return (part, *cur)

    total = 0.0
    for it0 in range(0, p["nt"], 10):
        part, *st = checkpoint(chunk, it0, min(p["nt"], it0 + 10), *leaves, *st, use_reentrant=False)
        total = total + part
    grads = dict(zip(names, torch.autograd.grad(total, leaves)))
    if case["prec"] != "f64":
        return {"misfit": total.item(), **grads}
    every = ("rho", "c11", "c13", "c15", "c33", "c35", "c55", "tau")
    return {"misfit": total.item(), "gradient": torch.stack([grads.get(k, torch.zeros_like(leaves[0])) for k in every])}


def exact(case, seed):
    call, p = case["call"], _problem(case, seed)
    if call == "gather":
        out = []
        for s in p:
            sim = _Exact(case, s["nx"], s["nz"], {k: t.double() for k, t in s["medium"].items()}, _taus(case),
                         s["sources"], s["receivers"], _rounded(case, s["nt"]))
            st, tr = sim.run(sim.start(), s["nt"])
            out.append({"traces": tr, **sim.fields(st)})
        return out
    wavelet = _rounded(case, p["nt"])
    if call == "gradient":
        return _exact_gradient(case, p, wavelet)
    sim = _Exact(case, p["nx"], p["nz"], {k: t.double() for k, t in p["medium"].items()}, _taus(case), p["sources"],
                 p["receivers"], wavelet)
    st, tr = sim.run(sim.start(p.get("state")), p["nt"])
    if call == "solve":
        return tr
    return sim.fields(st) if call == "leapfrog" else {"traces": tr, **sim.fields(st)}


def _rounded(case, nt):
    """The wavelet as the framework is given it."""
    return torch.as_tensor(_wavelet(nt), dtype=_dtype(case)).double().numpy()

"""Measured work of the wave-propagation engine: its schemes through the public Python entry points.

listed() holds one case or two per scheme and direction, draw(rng) draws from the same ranges.  A
state is what a modelling or inversion program keeps: an Engine with its model and shots set, the
observed data of an inversion, the arrays a survey call takes.  run() is one pass: a whole
forward, gradient or survey call, records or gradients whole.  exact() restates the same discrete
schemes in 64 bits with plain torch operations.

Kinds:
  acoustic        2-D velocity-pressure forward (orders 2 .. 16, constant or variable density,
                  aperture windows, uneven records, the reference's rounding order or not)
  gradient        its full-waveform gradient d misfit / d vp
  visco           2-D viscoacoustic forward, one memory variable
  visco_gradient  d misfit / d vp and d misfit / d (1/Q)
  viscoel         2-D visco-elastic forward, both record sets
  elastic         2-D isotropic elastic forward, free surface with topography or absorbing, vx and vz
  acoustic3d      3-D forward (orders 4 and 8)
  gradient3d      its gradient
  vti             survey call of the VTI pseudo-acoustic modeller
"""
import math

import numpy as np
import torch

from seismic_code_github_b200 import seisfd as S

PI32 = float(np.float32(3.1415926))
COEF = {1: [1.0], 2: [9 / 8, -1 / 24], 3: [75 / 64, -25 / 384, 3 / 640],
        4: [1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168],
        5: [19845 / 16384, -735 / 8192, 567 / 40960, -405 / 229376, 35 / 294912],
        8: [1.2340911, -1.0664985e-1, 2.3036367e-2, -5.3423856e-3, 1.0772712e-3, -1.6641888e-4, 1.7021711e-5,
            -8.5234642e-7]}
COEF = {r: [float(np.float32(v)) for v in c] for r, c in COEF.items()}


# ---- cases -------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: one shot of the reference program's own kind on a 251 x 251 model, records
        # to host memory; 1000 short steps, so latency counts
        dict(name="afd_one_shot", kind="acoustic", nx=251, nz=251, pml=50, order=16, shots=1, nt0=1000, nt1=1000,
             window=0, varden=False, exact=False, host=True),
        # a batched survey on the 512 x 2048 model: the largest 2-D work, records stay on the device
        dict(name="afd_survey", kind="acoustic", nx=2048, nz=512, pml=50, order=16, shots=64, nt0=200, nt1=200,
             window=0, varden=False, exact=False, host=False),
        # a line with aperture windows, uneven record lengths, variable density and odd sizes, 8th order
        dict(name="afd_windows_varden", kind="acoustic", nx=1501, nz=403, pml=40, order=8, shots=20, nt0=350, nt1=600,
             window=701, varden=True, exact=False, host=False),
        # the reference's rounding order, which the command-line programs run by default
        dict(name="afd_reference_order", kind="acoustic", nx=751, nz=351, pml=50, order=16, shots=8, nt0=400, nt1=400,
             window=0, varden=True, exact=True, host=True),
        # one inversion iteration's gradient on the 384 x 1536 model
        dict(name="fwi_gradient", kind="gradient", nx=1536, nz=384, pml=50, order=16, shots=16, nt0=400, nt1=400,
             varden=False),
        # viscoacoustic survey with uneven records on the 1024 x 1024 model
        dict(name="q_survey", kind="visco", nx=1024, nz=1024, pml=50, shots=16, nt0=160, nt1=240, exact=False),
        # viscoacoustic inversion gradient (vp and 1/Q)
        dict(name="q_gradient", kind="visco_gradient", nx=640, nz=360, pml=30, shots=8, nt0=300, nt1=400),
        # visco-elastic survey, P and S quality factors
        dict(name="viscoelastic_survey", kind="viscoel", nx=700, nz=500, pml=40, shots=8, nt0=200, nt1=260),
        # elastic survey under a free surface with topography
        dict(name="elastic_topography", kind="elastic", nx=1200, nz=403, pml=40, shots=8, nt0=250, nt1=300, free=True),
        # 3-D survey of two shots
        dict(name="cube_survey", kind="acoustic3d", nx=288, ny=272, nz=256, pml=32, order=8, shots=2, nt0=80, nt1=100,
             varden=False),
        # 3-D gradient
        dict(name="cube_gradient", kind="gradient3d", nx=136, ny=120, nz=100, pml=20, order=8, shots=2, nt0=130,
             nt1=150, varden=False),
        # VTI survey in the shipped card's geometry (300 x 300 model, 600 traces per shot)
        dict(name="vti_survey", kind="vti", nx=300, nz=300, traces=600, bound=50, top=0, shots=16, nt=600, exact=False),
    ]


def _lg(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, sizes over its whole range (log-uniform), odd ones among them, with the
    work of one pass below the largest listed case of the kind."""
    kind = rng.choice(["acoustic", "acoustic", "acoustic", "gradient", "visco", "visco_gradient", "viscoel", "elastic",
                       "acoustic3d", "gradient3d", "vti"])
    cap = {"acoustic": 1.6e10, "gradient": 5.0e9, "visco": 4.0e9, "visco_gradient": 9.0e8, "viscoel": 7.0e8,
           "elastic": 1.2e9, "acoustic3d": 7.0e9, "gradient3d": 8.0e8, "vti": 2.0e9}[kind]
    c = dict(kind=kind)
    if kind in ("acoustic3d", "gradient3d"):
        hi = 288 if kind == "acoustic3d" else 136
        c.update(nx=_lg(rng, 60, hi), ny=_lg(rng, 60, hi), nz=_lg(rng, 60, hi), pml=rng.randint(12, 32),
                 order=rng.choice([8, 8, 4]), varden=rng.random() < 0.3)
        cells = math.prod(c[a] + 2 * c["pml"] for a in ("nx", "ny", "nz"))
        shots, nt = rng.randint(1, 3), _lg(rng, 60, 150)
    elif kind == "vti":
        c.update(nx=_lg(rng, 120, 300), nz=_lg(rng, 120, 300), traces=_lg(rng, 120, 600), bound=rng.randint(20, 50),
                 top=rng.choice([0, 0, rng.randint(8, 40)]), exact=rng.random() < 0.25)
        cells = (c["traces"] + 2 * c["bound"]) * (c["nz"] + c["bound"] + c["top"])
        shots, nt = _lg(rng, 1, 16), _lg(rng, 300, 700)
    else:
        big = {"acoustic": (2048, 512), "gradient": (1536, 384), "visco": (1024, 1024), "visco_gradient": (640, 400),
               "viscoel": (700, 500), "elastic": (1200, 420)}[kind]
        c.update(nx=_lg(rng, 150, big[0]), nz=_lg(rng, 120, big[1]), pml=rng.randint(20, 50))
        cells = (c["nx"] + 2 * c["pml"]) * (c["nz"] + 2 * c["pml"])
        shots, nt = _lg(rng, 1, 64 if kind == "acoustic" else 16), _lg(rng, 150, 1000 if kind == "acoustic" else 400)
        if kind == "acoustic":
            window = rng.choice([0, 0, max(2 * c["pml"] + 40, int(c["nx"] * rng.uniform(0.4, 0.9)))])
            c.update(order=rng.choice([16, 16, 16, 10, 8, 4]), window=min(window, c["nx"]), varden=rng.random() < 0.4,
                     exact=rng.random() < 0.2, host=rng.random() < 0.5)
        elif kind == "gradient":
            c.update(order=rng.choice([16, 16, 8]), varden=rng.random() < 0.3)
        elif kind == "visco":
            c.update(exact=rng.random() < 0.25)
        elif kind == "elastic":
            c.update(free=rng.random() < 0.7)
    while cells * shots * nt > cap and shots > 1:
        shots -= 1
    nt = max(20, min(nt, int(cap / (cells * shots))))
    if kind == "vti":
        c.update(shots=shots, nt=nt)
    else:
        c.update(shots=shots, nt0=max(16, int(nt * rng.uniform(0.6, 1.0))), nt1=nt)
    return c


# ---- inputs ------------------------------------------------------------------------------------

def _ricker(nt, dt, f0, t0):
    """Zero-phase Ricker wavelet centred at t0 seconds."""
    a = (math.pi * f0 * (np.arange(nt) * dt - t0)) ** 2
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _layers(rng, nx, nz, vmin, vmax, ny=0):
    """Layers increasing with depth with a smooth lateral variation and (2-D) two smooth anomalies."""
    n = int(rng.integers(5, 12))
    cut = np.sort(rng.uniform(0.05, 0.95, n - 1)) * nz
    col = np.linspace(vmin, vmax, n)[np.searchsorted(cut, np.arange(nz), side="right")]
    k, p = rng.uniform(0.5, 3.0, 4) * 2 * np.pi, rng.uniform(0, 6.28, 4)
    x, z = np.arange(nx) / nx, np.arange(nz) / nz
    if ny:
        y = np.arange(ny) / ny
        lat = 1.0 + 0.03 * np.cos(k[0] * x[:, None] + p[0]) * np.cos(k[1] * y[None, :] + p[1])
        return np.clip(lat[:, :, None].astype(np.float32) * col.astype(np.float32), vmin * 0.96, vmax * 1.04)
    v = col[None, :] * (1.0 + 0.04 * np.cos(k[0] * x[:, None] + p[0]) * np.cos(k[1] * z[None, :] + p[1]))
    for _ in range(2):
        cx, cz = rng.uniform(0.2, 0.8, 2)
        v += rng.choice([-1, 1]) * 0.06 * vmin * np.exp(-((x[:, None] - cx) ** 2 + (z[None, :] - cz) ** 2) / 0.01)
    return np.clip(v, vmin * 0.95, vmax * 1.05).astype(np.float32)


def _pad(a, *pads):
    return np.ascontiguousarray(np.pad(a, pads, mode="edge"))


def _spread(c, n, margin):
    """Source columns of the shots, evenly spread."""
    return [int(margin + (i + 0.5) * n / c["shots"]) for i in range(c["shots"])]


def _lengths(c):
    """Record lengths of the shots, uneven between nt0 and nt1 (the survey's geometry: no seed in it)."""
    return [c["nt1"] - (i * 7919 + i * i * 31) % (c["nt1"] - c["nt0"] + 1) for i in range(c["shots"])]


def _observed(rng, shots, dt, d, f0, amp):
    """Observed records: a direct and a reflected arrival with hyperbolic moveout per trace."""
    out = []
    for s in shots:
        t = np.arange(s["nt"], dtype=np.float32)[None, :] * np.float32(dt)
        off = d * np.sqrt(sum((np.asarray(s["rec"][a]) - s["src"][a]) ** 2 for a in range(len(s["src"])))).astype(np.float32)
        rec = np.zeros((len(off), s["nt"]), np.float32)
        for v, h, g in ((rng.uniform(1500, 1700), 0.0, 1.0), (rng.uniform(1900, 2300), 300.0, 0.4)):
            arr = np.sqrt(off ** 2 + 4 * h * h) / v + s["t0"]
            b = (np.float32(math.pi * f0) * (t - arr[:, None].astype(np.float32))) ** 2
            rec += (g * amp / np.sqrt(1.0 + off / 50.0))[:, None].astype(np.float32) * (1 - 2 * b) * np.exp(-b)
        out.append(rec.reshape(-1))
    return np.concatenate(out)


def _inputs(c, seed):
    """Every input of a case, from the seed alone: grid numbers, padded models, shots, observed data."""
    rng = np.random.default_rng([int(seed), 77])
    kind, p = c["kind"], c.get("pml", 0)
    if kind == "vti":
        k = dict(dx=5.0, dt=5e-4, f0=30.0)
        vz = _layers(rng, c["nx"], c["nz"], 1500.0, 3400.0)
        e = (0.05 + 0.20 * (vz - 1400.0) / 2200.0).astype(np.float32)
        half = c["traces"] // 2
        cols = [1 + int((i + rng.uniform(0, 1)) * c["nx"] / c["shots"]) for i in range(c["shots"])]
        k.update(vz=vz, eps=e, delta=(0.45 * e).astype(np.float32), bounds=(c["bound"], c["bound"], c["top"], c["bound"]),
                 shots=[(s, 1, 1, s - half, s - half + c["traces"] - 1) for s in cols])
        return k
    k = dict(NX=c["nx"] + 2 * p, NZ=c["nz"] + 2 * p, nts=_lengths(c))
    if kind in ("acoustic3d", "gradient3d"):
        k.update(NY=c["ny"] + 2 * p, d=10.0, dt=1e-3, f0=25.0)
        vp = _layers(rng, c["nx"], c["nz"], 1600.0, 3800.0, ny=c["ny"])
        den = (1700.0 + 0.2 * vp).astype(np.float32) if c["varden"] else None
        k["vp"], k["den"] = (None if a is None else _pad(a, (p, p), (p, p), (p, p)) for a in (vp, den))
        k["shots"] = []
        for s, nt in enumerate(k["nts"]):
            sx, sy = p + int(rng.integers(c["nx"] // 4, 3 * c["nx"] // 4)), p + int(rng.integers(c["ny"] // 4, 3 * c["ny"] // 4))
            x0, y0 = max(p, sx - 32), max(p, sy - 32)
            rx, ry = np.meshgrid(np.arange(x0, min(x0 + 64, p + c["nx"])), np.arange(y0, min(y0 + 64, p + c["ny"])), indexing="ij")
            k["shots"].append(dict(src=(sx, sy, p + 2), rec=(rx.ravel(), ry.ravel(), np.full(rx.size, p + 2)), nt=nt,
                                   w=_ricker(nt, 1e-3, 25.0, 0.04), t0=0.04, x0=0, n=k["NX"]))
    else:
        f0 = {"acoustic": 25.0, "gradient": 20.0}.get(kind, 20.0)
        d = 10.0 if kind in ("acoustic", "gradient") else 5.0
        dt = 1e-3 if kind in ("acoustic", "gradient") else 5e-4
        k.update(d=d, dt=dt, f0=f0)
        vp = _layers(rng, c["nx"], c["nz"], 1500.0, 4000.0 if d == 10.0 else 3000.0)
        rho = (1600.0 + 0.25 * vp).astype(np.float32)
        pad = lambda a: _pad(a, (p, p), (p, p))  # noqa: E731
        k["vp"], k["den"] = pad(vp), pad(rho)
        if kind in ("acoustic", "gradient") and not c["varden"]:
            k["den"] = None
        if kind in ("visco", "visco_gradient", "viscoel"):
            q = (20.0 + 180.0 * (vp - vp.min()) / max(1.0, float(vp.max() - vp.min()))).astype(np.float32)
            cx, cz = rng.uniform(0.3, 0.7, 2) * (c["nx"], c["nz"])
            lens = (np.arange(c["nx"])[:, None] - cx) ** 2 + (np.arange(c["nz"])[None, :] - cz) ** 2 < (c["nz"] / 8) ** 2
            k["q"] = pad(np.where(lens, np.float32(20.0), q).astype(np.float32))
        if kind in ("viscoel", "elastic"):
            k["vs"] = (k["vp"] / np.float32(1.8)).astype(np.float32)
        if kind == "viscoel":
            k["qs"] = (np.float32(0.7) * k["q"]).astype(np.float32)
        top = None
        if kind == "elastic":
            k["rgau"] = 12
            if c["free"]:
                a, b = rng.uniform(0.5, 2.0), rng.uniform(0, 6.28)
                h = 6.0 + 5.0 * np.sin(2 * np.pi * a * np.arange(c["nx"]) / c["nx"] + b)
                top = p + np.round(np.pad(h, (p, p), mode="edge")).astype(np.int32)
                k["itopo"] = top
        n = c.get("window") or 0
        n = n + 2 * p if n else k["NX"]
        k["shots"] = []
        for sx, nt in zip(_spread(c, c["nx"], p), k["nts"]):
            x0 = min(max(0, sx - n // 2), k["NX"] - n)
            rx = np.arange(p, n - p)
            rz = np.full(rx.size, p + 2) if top is None else top[rx] + 1
            sz = p + 2 if top is None else int(top[sx]) + 3
            k["shots"].append(dict(src=(sx - x0, sz), rec=(rx, rz), nt=nt, w=_ricker(nt, dt, f0, 1.2 / f0), t0=1.2 / f0,
                                   x0=x0, n=n))
    if "gradient" in kind:
        amp = {"gradient": 4.0e5, "gradient3d": 1.0e5, "visco_gradient": 1.0e-6}[kind]
        k["obs"] = _observed(rng, k["shots"], k["dt"], k["d"], k["f0"], amp)
    return k


def prepare(case, seed):
    c, k = case, _inputs(case, seed)
    if c["kind"] == "vti":
        return dict(case=c, k=k)
    kind, p, three = c["kind"], c["pml"], c["kind"] in ("acoustic3d", "gradient3d")
    scheme = {"acoustic": S.ACOUSTIC_2D, "gradient": S.ACOUSTIC_2D, "visco": S.VISCOAC_2D, "visco_gradient": S.VISCOAC_2D,
              "viscoel": S.VISCOEL_2D, "elastic": S.ELASTIC_2D}.get(kind, S.ACOUSTIC_3D)
    e = S.Engine(scheme, k["NX"], k["NZ"], k["d"], k["d"], k["dt"], p, order=c.get("order", 10), ny=k.get("NY", 1),
                 dy=k["d"] if three else 0.0, flags=S.EXACT if c.get("exact") else 0, f0=k["f0"])
    if kind == "elastic":
        e.set_gauss_radius(k["rgau"])
        if c["free"]:
            e.set_free_surface(p)
            e.set_topography(k["itopo"])
        e.set_model_elastic(k["vp"], k["vs"], k["den"])
    elif kind == "viscoel":
        e.set_model_elastic(k["vp"], k["vs"], k["den"], k["q"], k["qs"])
    else:
        e.set_model(k["vp"], k["den"], k.get("q"))
    shots = []
    for s in k["shots"]:
        if three:
            shots.append(S.ShotSpec(s["src"][0], s["src"][2], s["rec"][0], s["rec"][2], s["w"], sy=s["src"][1], rec_y=s["rec"][1]))
        else:
            win = dict(ap_x0=s["x0"], ap_nx=s["n"]) if s["n"] != k["NX"] else {}
            shots.append(S.ShotSpec(s["src"][0], s["src"][1], s["rec"][0], s["rec"][1], s["w"], **win))
    e.set_shots(shots)
    st = dict(case=c, engine=e)
    if "gradient" in kind:
        shape = k["vp"].shape
        st["obs"] = torch.from_numpy(k["obs"]).cuda()
        st["misfit"] = torch.zeros(1, device="cuda")
        st["grad_vp"] = torch.zeros(shape, device="cuda")
        st["grad_invq"] = torch.zeros(shape, device="cuda") if kind == "visco_gradient" else None
    elif kind not in ("viscoel", "elastic") and not c.get("host"):
        st["records"] = torch.zeros(e.record_size(), device="cuda")
    return st


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "vti":
        k = state["k"]
        return S.vti_forward(k["vz"], k["eps"], k["delta"], k["dx"], k["dx"], k["dt"], k["f0"], c["nt"], k["bounds"],
                             k["shots"], exact=c["exact"])[0]
    e = state["engine"]
    if "gradient" in kind:
        q = state["grad_invq"]
        e.gradient_device(state["obs"].data_ptr(), state["misfit"].data_ptr(), state["grad_vp"].data_ptr(),
                          None if q is None else q.data_ptr())
        out = dict(misfit=state["misfit"], grad_vp=state["grad_vp"])
        return out if q is None else dict(out, grad_invq=q)
    if kind == "viscoel":
        return dict(szz=e.forward(), sxx=e.records(S.FIELD_P))
    if kind == "elastic":
        return dict(vx=e.forward(), vz=e.records(S.FIELD_VZ))
    if c.get("host"):
        return e.forward()
    e.forward_device(state["records"].data_ptr())
    return state["records"]


# bytes and operations per grid point and step: each state field read and written once, each model
# field read once; the gradient: one forward and one adjoint pass (D_k written and read once)
_WORK = {"acoustic": (28, 132), "gradient": (28 + 40 + 4, 270), "visco": (40, 110), "visco_gradient": (40 + 60 + 8, 240),
         "viscoel": (92, 260), "elastic": (60, 200), "acoustic3d": (36, 100), "gradient3d": (36 + 52, 210), "vti": (36, 80)}


def work(case):
    c, (b, f) = case, _WORK[case["kind"]]
    p = c.get("pml", 0)
    if c["kind"] == "vti":
        steps = c["nt"] + 140
        cells = (c["traces"] + 2 * c["bound"] - 2) * (c["nz"] + c["bound"] + c["top"] - 2)
        rec = c["shots"] * c["traces"] * c["nt"] * 4
        return dict(bytes=cells * steps * c["shots"] * b + rec, flops=cells * steps * c["shots"] * f)
    n = (c.get("window") or c["nx"]) + 2 * p
    cells = n * (c["nz"] + 2 * p) * ((c["ny"] + 2 * p) if "ny" in c else 1)
    if c.get("varden"):
        b += 4
    if c["kind"] in ("acoustic", "gradient", "gradient3d", "acoustic3d"):
        f = f * (c["order"] / (16 if c["kind"] in ("acoustic", "gradient") else 8))
    steps = 0.5 * (c["nt0"] + c["nt1"]) * c["shots"]
    nrec = 64 * 64 if "ny" in c else (c.get("window") or c["nx"])
    return dict(bytes=cells * steps * b + 4 * nrec * steps, flops=cells * steps * f)


# ---- 64-bit restatement ------------------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev()).double()


def _f(v):
    return float(np.float32(v))


class _Acoustic:
    """Velocity-pressure scheme on [shot, x, (y,) z]: forward step and its transpose."""

    def __init__(self, c, k, s0):
        p, R = c["pml"], c["order"] // 2
        self.R, self.C, self.dt, self.d = R, COEF[R], _f(k["dt"]), _f(k["d"])
        x0, n = s0["x0"], s0["n"]
        self.vp = _t(k["vp"][x0:x0 + n])
        self.den = _t(k["den"][x0:x0 + n]) if k["den"] is not None else torch.full_like(self.vp, 2400.0)
        dims = self.vp.shape
        ab = torch.ones_like(self.vp)
        for ax in reversed(range(len(dims))):  # x wins over y over z
            q = torch.arange(dims[ax], device=ab.device)
            q = torch.where(q < p, p - q - 1, torch.where(q >= dims[ax] - p, q - dims[ax] + p, -1))
            tap = (1 - 0.38 * q.double() ** 2 / (1.0 * p * p)).float().double()
            view = [1] * len(dims)
            view[ax] = -1
            ab = torch.where((q >= 0).view(view), tap.view(view), ab)
        self.ab = ab
        self.dims, self.nd = dims, len(dims)
        self.K = self.den * self.vp ** 2 * self.dt
        self.b = self.dt / (self.den * self.d)

    def inner(self, u):
        for a in range(self.nd):
            u = u.narrow(u.dim() - self.nd + a, self.R, self.dims[a] - 2 * self.R)
        return u

    def _cut(self, u, ax, o):
        for a in range(self.nd):
            u = u.narrow(1 + a, self.R + (o if a == ax else 0), self.dims[a] - 2 * self.R)
        return u

    def diff(self, u, ax, fwd):
        """Staggered difference on the updated cells: forward (velocities) or backward (pressure)."""
        acc = None
        for m, cm in enumerate(self.C, 1):
            t = self._cut(u, ax, m if fwd else m - 1) - self._cut(u, ax, 1 - m if fwd else -m)
            acc = t.mul_(cm) if acc is None else acc.add_(t, alpha=cm)
        return acc

    def diff_t(self, y, ax, fwd, out):
        """out += transpose of diff."""
        for m, cm in enumerate(self.C, 1):
            self._cut(out, ax, m if fwd else m - 1).add_(y, alpha=cm)
            self._cut(out, ax, 1 - m if fwd else -m).add_(y, alpha=-cm)

    def state(self, ns):
        return [torch.zeros((ns,) + tuple(self.dims), dtype=torch.float64, device=self.vp.device) for _ in range(1 + self.nd)]

    def step(self, st, src, w, keep=None):
        P = st[0]
        P[src] -= self.dt * self.den[src[1:]] * self.vp[src[1:]] * w
        div = None
        for a in range(self.nd):
            self.inner(st[1 + a]).sub_(self.diff(P, a, True).mul_(self.inner(self.b)))
        for a in range(self.nd):
            t = self.diff(st[1 + a], a, False).div_(self.d)
            div = t if div is None else div.add_(t)
        if keep is not None:
            keep.append(div.clone())
        self.inner(P).sub_(div.mul_(self.inner(self.K)))
        for u in st:
            u.mul_(self.ab)

    def adjoint(self, st, div, gK):
        """Transpose of step, from the sponge back to the source; gK -= nu div."""
        for u in st:
            u.mul_(self.ab)
        P = st[0]
        gK.sub_((self.inner(P) * div).sum(0))
        kp = self.inner(P) * (self.inner(self.K) / self.d)
        for a in range(self.nd):
            self.diff_t(-kp, a, False, st[1 + a])
        for a in range(self.nd):
            self.diff_t(-(self.inner(st[1 + a]) * self.inner(self.b)), a, True, P)


def _src(shots):
    cols = list(zip(*[s["src"] for s in shots]))
    dev = _dev()
    return (torch.arange(len(shots), device=dev),) + tuple(torch.tensor(v, device=dev) for v in cols)


def _wave(shots, nt):
    w = np.zeros((len(shots), nt))
    for i, s in enumerate(shots):
        w[i, :s["nt"]] = s["w"]
    return _t(w)


def _rec_index(shots):
    dev = _dev()
    idx = [torch.cat([torch.full((len(s["rec"][0]),), i, device=dev, dtype=torch.long) for i, s in enumerate(shots)])]
    for a in range(len(shots[0]["rec"])):
        idx.append(torch.cat([torch.as_tensor(np.asarray(s["rec"][a]), device=dev).long() for s in shots]))
    return tuple(idx)


def _flat(shots, rec):
    """[receiver of all shots, nt_max] to the flat record layout (each shot its own nt)."""
    out, o = [], 0
    for s in shots:
        n = len(s["rec"][0])
        out.append(rec[o:o + n, :s["nt"]].reshape(-1))
        o += n
    return torch.cat(out)


def _exact_acoustic(c, k):
    groups = {}
    for i, s in enumerate(k["shots"]):
        groups.setdefault((s["x0"], s["n"]), []).append(i)
    out = [None] * len(k["shots"])
    for ids in groups.values():
        shots = [k["shots"][i] for i in ids]
        m, nt = _Acoustic(c, k, shots[0]), max(s["nt"] for s in shots)
        st, src, w, ri = m.state(len(shots)), _src(shots), _wave(shots, nt), _rec_index(shots)
        rec = torch.zeros(len(ri[0]), nt, dtype=torch.float64, device=_dev())
        for t in range(nt):
            m.step(st, src, w[:, t])
            rec[:, t] = st[0][ri]
        o = 0
        for i, s in zip(ids, shots):
            n = len(s["rec"][0])
            out[i] = rec[o:o + n, :s["nt"]].reshape(-1)
            o += n
    return torch.cat(out)


def _residual(shots, rec, obs, nt):
    """Residuals [receiver, nt_max] (zero past a shot's record) and the misfit."""
    res, o, q, mis = torch.zeros_like(rec), 0, 0, 0.0
    for s in shots:
        n = len(s["rec"][0])
        r = rec[o:o + n, :s["nt"]] - obs[q:q + n * s["nt"]].view(n, s["nt"])
        res[o:o + n, :s["nt"]] = r
        mis = mis + 0.5 * (r ** 2).sum()
        o, q = o + n, q + n * s["nt"]
    return res, mis


def _exact_gradient(c, k):
    shots = k["shots"]
    m, nt = _Acoustic(c, k, shots[0]), max(s["nt"] for s in shots)
    src, w, ri = _src(shots), _wave(shots, nt), _rec_index(shots)
    C = max(1, int(math.sqrt(nt)))
    st, cks = m.state(len(shots)), []
    rec = torch.zeros(len(ri[0]), nt, dtype=torch.float64, device=_dev())
    for t in range(nt):
        if t % C == 0:
            cks.append([u.clone() for u in st])
        m.step(st, src, w[:, t])
        rec[:, t] = st[0][ri]
    res, mis = _residual(shots, rec, _t(k["obs"]), nt)
    adj, gK, gs = m.state(len(shots)), torch.zeros_like(m.inner(m.vp)), torch.zeros_like(m.vp)
    for j in reversed(range(len(cks))):
        st, keep = cks.pop(), []
        a, b = j * C, min(nt, j * C + C)
        for t in range(a, b):
            m.step(st, src, w[:, t], keep)
        for t in reversed(range(a, b)):
            adj[0].index_put_(ri, res[:, t], accumulate=True)
            m.adjoint(adj, keep.pop(), gK)
            gs.index_put_(src[1:], -adj[0][src] * m.dt * m.den[src[1:]] * w[:, t], accumulate=True)
    m.inner(gs).add_(gK * m.inner(2.0 * m.den * m.vp * m.dt))
    return dict(misfit=mis.reshape(1), grad_vp=gs)


def _rsg(u, xdir, flag, h):
    """Rotated-staggered derivative of [shot, x, z] with zeros outside the grid."""
    X, Z = u.shape[1:]
    up = torch.nn.functional.pad(u, (5, 5, 5, 5))
    g = lambda dk, di: up[:, 5 + di:5 + di + X, 5 + dk:5 + dk + Z]  # noqa: E731
    acc = None
    for m, am in enumerate(COEF[5]):
        hi, lo = (m, -1 - m) if flag == 0 else (1 + m, -m)
        t = g(hi, hi) - g(lo, lo)
        s = g(lo, hi) - g(hi, lo)
        t = t.add_(s) if xdir else t.sub_(s)
        acc = t.mul_(am) if acc is None else acc.add_(t, alpha=am)
    return acc.mul_(h)


def _cosine(n, p, d):
    """Sponge factors along one axis of n cells: integer points, and the half points of the stress."""
    r = math.acos(_f(1e-3)) / (p * d)
    a, b = torch.ones(n, dtype=torch.float64), torch.ones(n, dtype=torch.float64)
    for i in range(p + 1):
        q = (p - i) * d
        a[i] *= math.cos(r * q)
        b[i] *= 1.0 if i == p else math.cos(r * (q - d / 2))
        a[n - 1 - i] *= math.cos(r * q)
        b[n - 1 - i] *= math.cos(r * (q + d / 2))
    return a.to(_dev()), b.to(_dev())


def _blanch(k, rho, q):
    """tau ratio of Blanch's method and 1 / tau_sigma."""
    flow, fup = 4.0 * PI32, 2.5 * _f(k["f0"]) * 2.0 * PI32
    tss = 1.0 / ((fup - flow) / 2.0)
    num = math.log(tss ** 2 * fup ** 2 + 1) - math.log(tss ** 2 * flow ** 2 + 1)
    f = lambda w: math.atan(w * tss) - w * tss / (1 + tss ** 2 * w ** 2)  # noqa: E731
    kap = num / (f(fup) - f(flow)) * (20.0 / 18.0)
    return 1.0 + kap / q, kap, 1.0 / tss


def _mean_rho(rho):
    r = rho.clone()
    r[:-1, :-1] = 0.25 * (rho[:-1, :-1] + rho[:-1, 1:] + rho[1:, 1:] + rho[1:, :-1])
    # the average runs in place: a cell's neighbours above and to the right are still the given ones
    r[:, -1] = r[:, -2]
    r[-1, :] = r[-2, :]
    return r


def _gauss(X, Z, shots, sigma, rad, even_shift):
    """Normalised Gaussian source stamps [shot, x, z]."""
    out = torch.zeros(len(shots), X, Z, dtype=torch.float64, device=_dev())
    n = min(rad, 30)
    o = torch.arange(-n + 1, n, dtype=torch.float64, device=_dev())
    g = torch.exp(-(o[:, None] ** 2 + o[None, :] ** 2) / (2 * sigma ** 2))
    g = g / g.sum()
    for i, s in enumerate(shots):
        cx = s["src"][0] - (1 if even_shift and X % 2 == 0 else 0)
        cz = s["src"][1] - (1 if even_shift and Z % 2 == 0 else 0)
        x0, x1, z0, z1 = max(0, cx - n + 1), min(X, cx + n), max(0, cz - n + 1), min(Z, cz + n)
        out[i, x0:x1, z0:z1] = g[x0 - cx + n - 1:x1 - cx + n - 1, z0 - cz + n - 1:z1 - cz + n - 1]
    return out


class _Visco:
    """Viscoacoustic step on split fields and its transpose.  Fields: vx vz sx sz sr rx rz rr."""

    def __init__(self, c, k):
        p, d = c["pml"], _f(k["d"])
        self.dt, self.h = _f(k["dt"]), 0.5 / d
        self.vp, rho = _t(k["vp"]), _mean_rho(_t(k["den"]))
        tau, self.kap, rt = _blanch(k, rho, _t(k["q"]))
        self.lam, self.b = rho * self.vp ** 2, 1.0 / rho
        self.p1, self.p2, self.f = self.lam * tau, self.lam * (tau - 1.0), -self.dt * rt
        X, Z = self.vp.shape
        ax, bx = _cosine(X, p, d)
        az, bz = _cosine(Z, p, d)
        self.ax, self.bx, self.az, self.bz = ax[:, None], bx[:, None], az[None, :], bz[None, :]
        self.stamp = _gauss(X, Z, k["shots"], 1.5, 30, True) * (self.dt / d ** 2)

    def state(self):
        return [torch.zeros_like(self.stamp) for _ in range(8)]

    def step(self, st, w, keep=None):
        vx, vz, sx, sz, sr, rx, rz, rr = st
        sig = sx + sz + sr
        vx.add_(_rsg(sig, True, 0, self.h).mul_(self.dt * self.b)).mul_(self.ax)
        vz.add_(_rsg(sig, False, 0, self.h).mul_(self.dt * self.b)).mul_(self.az)
        d1, d4 = _rsg(vx, True, 1, self.h), _rsg(vz, False, 1, self.h)
        if keep is not None:
            keep.append((d1, d4))
        r = rx + rz + rr
        sx.add_(self.dt * self.p1 * d1).mul_(self.bx).add_(w[:, None, None] * self.stamp)
        sz.add_(self.dt * self.p1 * d4).mul_(self.bz)
        sr.add_(r, alpha=self.dt)
        rx.add_(self.f * self.p2 * d1).mul_(self.bx)
        rz.add_(self.f * self.p2 * d4).mul_(self.bz)
        rr.add_(r, alpha=self.f)
        return sx + sz + sr

    def adjoint(self, st, kept, g1, g2):
        vx, vz, sx, sz, sr, rx, rz, rr = st
        d1, d4 = kept
        sx.mul_(self.bx), sz.mul_(self.bz), rx.mul_(self.bx), rz.mul_(self.bz)
        g1.add_(((sx * d1 + sz * d4) * self.dt).sum(0))
        g2.add_(((rx * d1 + rz * d4) * self.f).sum(0))
        # the memory sum of the previous step feeds sr and rr
        ar = self.dt * sr + self.f * rr
        a1 = self.dt * self.p1 * sx + self.f * self.p2 * rx
        a4 = self.dt * self.p1 * sz + self.f * self.p2 * rz
        for u in (rx, rz, rr):
            u.add_(ar)
        vx.sub_(_rsg(a1, True, 0, self.h)).mul_(self.ax)
        vz.sub_(_rsg(a4, False, 0, self.h)).mul_(self.az)
        asig = -_rsg(vx * (self.dt * self.b), True, 1, self.h) - _rsg(vz * (self.dt * self.b), False, 1, self.h)
        for u in (sx, sz, sr):
            u.add_(asig)


def _exact_visco(c, k):
    m, shots = _Visco(c, k), k["shots"]
    nt = max(s["nt"] for s in shots)
    w, ri, st = _wave(shots, nt), _rec_index(shots), m.state()
    rec = torch.zeros(len(ri[0]), nt, dtype=torch.float64, device=_dev())
    for t in range(nt):
        rec[:, t] = m.step(st, w[:, t])[ri]
    return _flat(shots, rec)


def _exact_visco_gradient(c, k):
    m, shots = _Visco(c, k), k["shots"]
    nt = max(s["nt"] for s in shots)
    w, ri, st = _wave(shots, nt), _rec_index(shots), m.state()
    C, cks = max(1, int(math.sqrt(nt))), []
    rec = torch.zeros(len(ri[0]), nt, dtype=torch.float64, device=_dev())
    for t in range(nt):
        if t % C == 0:
            cks.append([u.clone() for u in st])
        rec[:, t] = m.step(st, w[:, t])[ri]
    res, mis = _residual(shots, rec, _t(k["obs"]), nt)
    adj, g1, g2 = m.state(), torch.zeros_like(m.p1), torch.zeros_like(m.p1)
    inj = torch.zeros_like(adj[0])
    for j in reversed(range(len(cks))):
        st, keep = cks.pop(), []
        a, b = j * C, min(nt, j * C + C)
        for t in range(a, b):
            m.step(st, w[:, t], keep)
        for t in reversed(range(a, b)):
            inj.zero_().index_put_(ri, res[:, t], accumulate=True)
            for u in adj[2:5]:
                u.add_(inj)
            m.adjoint(adj, keep.pop(), g1, g2)
    gvp = (g1 * m.p1 + g2 * m.p2) * 2.0 / m.vp
    return dict(misfit=mis.reshape(1), grad_vp=gvp, grad_invq=(g1 + g2) * m.lam * m.kap)


def _exact_viscoel(c, k):
    p, d, dt, shots = c["pml"], _f(k["d"]), _f(k["dt"]), k["shots"]
    h = 0.5 / d
    vp, vs, rho = _t(k["vp"]), _t(k["vs"]), _mean_rho(_t(k["den"]))
    tp, _, rt = _blanch(k, rho, _t(k["q"]))
    ts = _blanch(k, rho, _t(k["qs"]))[0]
    mu, lm, f = rho * vs ** 2, rho * vp ** 2, -dt * rt
    q1, q2, q3 = lm * tp, lm * tp - 2 * mu * ts, mu * ts
    m1, m2, m3 = lm * (tp - 1), lm * (tp - 1) - 2 * mu * (ts - 1), mu * (ts - 1)
    X, Z = vp.shape
    (ax, bx), (az, bz) = _cosine(X, p, d), _cosine(Z, p, d)
    ax, bx, az, bz = ax[:, None], bx[:, None], az[None, :], bz[None, :]
    stamp = _gauss(X, Z, shots, 1.5, 30, True) * (dt / d ** 2)
    zero = lambda n: [torch.zeros_like(stamp) for _ in range(n)]  # noqa: E731
    vxx, vxz, vzx, vzz = zero(4)
    s, r = {a: zero(3) for a in ("xx", "zz", "xz")}, {a: zero(3) for a in ("xx", "zz", "xz")}
    nt = max(q["nt"] for q in shots)
    w, ri = _wave(shots, nt), _rec_index(shots)
    rec = torch.zeros(2, len(ri[0]), nt, dtype=torch.float64, device=_dev())
    sxx, szz, sxz = zero(3)
    for t in range(nt):
        vxx.add_(_rsg(sxx, True, 0, h).mul_(dt / rho)).mul_(ax)
        vxz.add_(_rsg(sxz, False, 0, h).mul_(dt / rho)).mul_(az)
        vzx.add_(_rsg(sxz, True, 0, h).mul_(dt / rho)).mul_(ax)
        vzz.add_(_rsg(szz, False, 0, h).mul_(dt / rho)).mul_(az)
        vx, vz = vxx + vxz, vzx + vzz
        d1, d2, d3, d4 = _rsg(vx, True, 1, h), _rsg(vz, True, 1, h), _rsg(vx, False, 1, h), _rsg(vz, False, 1, h)
        src = w[:, t, None, None] * stamp
        for a, cx, ux, cz, uz, mx, mz in (("xx", q1, d1, q2, d4, m1, m2), ("zz", q2, d1, q1, d4, m2, m1),
                                          ("xz", q3, d2, q3, d3, m3, m3)):
            old = r[a][0] + r[a][1] + r[a][2]
            s[a][0].add_(dt * cx * ux).mul_(bx)
            s[a][1].add_(dt * cz * uz).mul_(bz)
            s[a][2].add_(old, alpha=dt)
            if a != "xz":
                s[a][0].add_(src)
            r[a][0].add_(f * mx * ux).mul_(bx)
            r[a][1].add_(f * mz * uz).mul_(bz)
            r[a][2].add_(old, alpha=f)
        sxx, szz, sxz = (s[a][0] + s[a][1] + s[a][2] for a in ("xx", "zz", "xz"))
        rec[0, :, t], rec[1, :, t] = szz[ri], sxx[ri]
    return dict(szz=_flat(shots, rec[0]), sxx=_flat(shots, rec[1]))


def _exact_elastic(c, k):
    """Free-surface elastic scheme (the absorbing mode's top sponge is smoothed by a serial chain of a
    few hundred million dependent additions and has no 64-bit value here)."""
    p, d, dt, shots = c["pml"], _f(k["d"]), _f(k["dt"]), k["shots"]
    vp, vs, rho = _t(k["vp"]), _t(k["vs"]), _t(k["den"])
    X, Z = vp.shape
    top = torch.as_tensor(k["itopo"], device=_dev()).long() - 1  # 0-based surface row
    mu = rho * vs ** 2
    la = rho * vp ** 2 - 2 * mu
    b1 = 1.0 / _mean_rho(rho)
    b1e = torch.cat([b1[:, :1], 0.5 * (b1[:, 1:] + b1[:, :-1])], 1)
    avx = lambda u: torch.cat([0.5 * (u[:-1] + u[1:]), u[-1:]], 0)  # noqa: E731
    b2e, lam, lm2 = avx(1.0 / rho), avx(la), avx(la + 2 * mu)
    ms = torch.cat([0.5 * (mu[:, 1:] + mu[:, :-1]), mu[:, -1:]], 1)
    mue = ms.clone()
    mue[:-1, 1:] = 4.0 / (1 / ms[:-1, 1:] + 1 / ms[1:, 1:] + 1 / ms[1:, :-1] + 1 / ms[:-1, :-1])
    z = torch.arange(Z, device=_dev())[None, :]
    row = torch.maximum(z, top[:, None])  # rows above the surface take the surface row's values
    b2e, b1e, lam, lm2, mue = (torch.gather(u, 1, row.expand(X, Z)) for u in (b2e, b1e, lam, lm2, mue))
    upd = (z >= top[:, None]).double()
    dist = z - top[:, None]
    terms = (dist.clamp(1, 5), torch.where(dist >= 4, 5, dist.clamp(min=0) + 1))
    (ax, bx), (az, bz) = _cosine(X, p, d), _cosine(Z, p, d)
    az[:Z // 2], bz[:Z // 2] = 1.0, 1.0  # no top sponge
    one = torch.ones((), dtype=torch.float64, device=_dev())
    ax, bx = (torch.where(upd > 0, u[:, None], one) for u in (ax, bx))
    az, bz = az[None, :], bz[None, :]
    g = _gauss(X, Z, shots, 2.0, k["rgau"], False) * (dt / d ** 2)
    below = torch.tensor([s["src"][1] > int(top[s["src"][0]]) for s in shots], device=_dev()).double()

    def dx(u, flag):
        up = torch.nn.functional.pad(u, (0, 0, 5, 5))
        return sum(a * (up[:, 5 + (m if flag == 0 else 1 + m):][:, :X] - up[:, 5 + (-1 - m if flag == 0 else -m):][:, :X])
                   for m, a in enumerate(COEF[5]))

    def dz(u, flag):
        up = torch.nn.functional.pad(u, (5, 5))
        t = [up[..., 5 + (m if flag == 0 else 1 + m):][..., :Z] - up[..., 5 + (-1 - m if flag == 0 else -m):][..., :Z]
             for m in range(5)]
        out = None
        for n in range(1, 6):
            v = sum(a * t[m] for m, a in enumerate(COEF[n]))
            out = v if out is None else torch.where(terms[flag] == n, v, out)
        return out

    st = [torch.zeros_like(g) for _ in range(10)]
    vxx, vxz, vzx, vzz, xxx, xxz, zzx, zzz, xzx, xzz = st
    nt = max(s["nt"] for s in shots)
    w, ri = _wave(shots, nt), _rec_index(shots)
    rec = torch.zeros(2, len(ri[0]), nt, dtype=torch.float64, device=_dev())
    ix, wet = torch.arange(X, device=_dev()), top >= 1
    cols = ix[wet]
    air = (z <= top[:, None])[None]
    kq = dt / d
    ratio = (lam / lm2)[ix[:-1], top[:-1]]
    for t in range(nt):
        sxx, szz, sxz = xxx + xxz, zzx + zzz, xzx + xzz
        vxx.add_(kq * b2e * upd * dx(sxx, 0)).mul_(ax)
        vxz.add_(kq * b2e * upd * dz(sxz, 0)).mul_(az)
        vzx.add_(kq * b1e * upd * dx(sxz, 1)).mul_(bx)
        vzz.add_(kq * b1e * upd * dz(szz, 1)).mul_(bz)
        vx, vz = vxx + vxz, vzx + vzz
        src = w[:, t, None, None] * g
        d1, d2, d3, d4 = dx(vx, 1), dz(vz, 0), dx(vz, 0), dz(vx, 1)
        xxx.add_(kq * lm2 * upd * d1).mul_(bx).add_(src * below[:, None, None])
        xxz.add_(kq * lam * upd * d2).mul_(az)
        zzx.add_(kq * lam * upd * d1).mul_(bx).masked_fill_(air, 0.0).add_(src)
        zzz.add_(kq * lm2 * upd * d2).mul_(az).masked_fill_(air, 0.0)
        xzx.add_(kq * mue * upd * d3).mul_(ax)
        xzz.add_(kq * mue * upd * d4).mul_(bz)
        rec[0, :, t], rec[1, :, t] = vx[ri], vz[ri]
        for u in (xzx, xzz):  # image row above the surface
            u[:, cols, top[cols] - 1] = -u[:, cols, top[cols]]
        e, h = ix[:-1][wet[:-1]], top[:-1][wet[:-1]]
        for a, b in ((vxx, vzx), (vxz, vzz)):  # vz above the surface, read by the next stress update
            b[:, e, h - 1] = b[:, e, h] + ratio[wet[:-1]] * (a[:, e + 1, h] - a[:, e, h])
    return dict(vx=_flat(shots, rec[0]), vz=_flat(shots, rec[1]))


def _exact_vti(c, k):
    nxl, nxr, nzu, nzd = k["bounds"]
    rng, shots, dev = c["traces"], k["shots"], _dev()
    nx, nz = rng + nxl + nxr - 2, c["nz"] + nzu + nzd - 2
    dx, dt, f0 = _f(k["dx"]), _f(k["dt"]), _f(k["f0"])

    def taylor(first):
        i = np.arange(1, 6, dtype=np.float64)
        a = np.stack([i ** q / math.factorial(q) for q in ((1, 3, 5, 7, 9) if first else (2, 4, 6, 8, 10))], 1)
        return [float(v) for v in 0.5 * np.linalg.inv(a)[0]]

    cE, c1 = taylor(False), taylor(True)
    # windows [shot, z, x]
    m = {a: _t(k[a]) for a in ("vz", "eps", "delta")}
    V = torch.zeros(len(shots), nz, nx, dtype=torch.float64, device=dev)
    E, D = torch.zeros_like(V), torch.zeros_like(V)
    jj = (torch.arange(nz, device=dev) - nzu).clamp(0, c["nz"] - 1)
    ii = torch.arange(nx, device=dev) - nxl
    ins = (ii[None, :] >= 0) & (ii[None, :] < rng) & (torch.arange(nz, device=dev)[:, None] >= nzu) & \
        (torch.arange(nz, device=dev)[:, None] < nzu + c["nz"])
    for s, (nsx, nsz, nrz, xmin, _) in enumerate(shots):
        io = (ii.clamp(0, rng - 1) + xmin).clamp(0, c["nx"] - 1)
        V[s] = m["vz"][io][:, jj].T
        for u, a in ((E, "eps"), (D, "delta")):
            u[s] = torch.where(ins, m[a][io][:, jj].T, torch.zeros((), dtype=torch.float64, device=dev))
            u[s, :nsz + nzu + 6] = 0.0
    i, j = torch.arange(1, nx + 1, device=dev)[None, :], torch.arange(1, nz + 1, device=dev)[:, None]
    left, right = i <= nxl, i >= nx - nxr + 1
    side = (left | right).expand(nz, nx)
    topz, botz = j <= nzu, j >= nz - nzd + 1
    vert = ((topz | botz).expand(nz, nx)) & ~side
    vn2, vx2 = V ** 2 * (1 + 2 * D), V ** 2 * (1 + 2 * E)
    L = math.log(1.0 / _f(1e-3))

    def damp(v, axis, thick):
        return 1.5 * v / thick * (axis / thick) ** 2 * L, 1.5 * v / thick * 2 * axis / thick ** 2 * L

    thx = torch.where(left, float(nxl), float(nxr)).double().clamp(min=1) * dx
    dX, ddX = damp(vx2.sqrt(), torch.where(left, i - (nxl + 1), i - (nx - nxr)).double() * dx, thx)
    thz = torch.where(topz, float(nzu), float(nzd)).double().clamp(min=1) * dx
    dZ, ddZ = damp(V, torch.where(topz, j - (nzu + 1), j - (nz - nzd)).double() * dx, thz)

    def d2(u, ax):
        n = u.shape[ax]
        up = torch.nn.functional.pad(u, (5, 5) if ax == 2 else (0, 0, 5, 5))
        return sum(a * (up.narrow(ax, 5 + q, n) + up.narrow(ax, 5 - q, n) - 2 * u) for q, a in enumerate(cE, 1)) / dx ** 2

    def d1(u, ax):
        n = u.shape[ax]
        up = torch.nn.functional.pad(u, (5, 5) if ax == 2 else (0, 0, 5, 5))
        return sum(a * (up.narrow(ax, 5 + q, n) - up.narrow(ax, 5 - q, n)) for q, a in enumerate(c1, 1)) / dx

    z0 = lambda n: [torch.zeros_like(V) for _ in range(n)]  # noqa: E731
    U, Q = z0(2), z0(2)  # current, old
    # split fields (a1, t2, a2, a3), current and old, of u on the sides, of u above / below, of q on the sides
    F = {a: [z0(4), z0(4)] for a in ("ux", "uz", "qx")}

    def split(f, d, dd, k2, s2, s1):
        """The damped recurrences of one split set; returns the new (a1, t2, a2)."""
        (a1, t2, a2, _), (a1o, t2o, _, _) = f
        q = 1 + 2 * d * dt
        n1 = (a1 * (2 + 2 * d * dt - d ** 2 * dt ** 2) - a1o + k2 * s2) / q
        nt = (t2 * (2 + 2 * d * dt - d ** 2 * dt ** 2) - t2o - k2 * dd * s1) / q
        return n1, nt, a2 * (1 - d * dt) + nt * dt

    nwt = int(math.floor((2 * 0.07) / dt + 0.5)) + 1
    half = int(math.floor((nwt - 1) / 2.0 + 0.5))
    rec = torch.zeros(len(shots), rng, c["nt"], dtype=torch.float64, device=dev)
    sidx = torch.arange(len(shots), device=dev)
    sx = torch.tensor([s[0] - s[3] + nxl - 1 for s in shots], device=dev)
    sz = torch.tensor([s[1] + nzu - 1 for s in shots], device=dev)
    rr = shots[0][2] + nzu
    low = rr < 6
    rr = 6 if low else rr
    for it in range(1, c["nt"] + half + 1):
        if it <= nwt:
            b = PI32 * f0 * (it - 0.07 / dt) * dt
            U[0][sidx, sz, sx] += math.exp(-b * b) * (1 - 2 * b * b)
        u, q = U[0], Q[0]
        sxu, sxq, szu = d2(u, 2), d2(q, 2), d2(u, 1)
        s2, s1, sz1 = sxu + sxq, d1(u, 2) + d1(q, 2), d1(u, 1)
        new = {}
        n = split(F["ux"], dX, ddX, vn2 * dt ** 2, s2, s1)
        a3 = 2 * F["ux"][0][3] - F["ux"][1][3] + V ** 2 * dt ** 2 * szu
        new["ux"] = [t * side for t in (*n, a3)]
        n = split(F["uz"], dZ, ddZ, V ** 2 * dt ** 2, szu, sz1)
        a3 = 2 * F["uz"][0][3] - F["uz"][1][3] + vn2 * dt ** 2 * s2
        new["uz"] = [t * vert for t in (*n, a3)]
        n = split(F["qx"], dX, ddX, (vx2 - vn2) * dt ** 2, s2, s1)
        new["qx"] = [t * side for t in n] + [torch.zeros((), dtype=torch.float64, device=dev)]
        un = 2 * u - U[1] + dt ** 2 * V ** 2 * ((1 + 2 * D) * s2 + szu)
        un = torch.where(side, new["ux"][0] + new["ux"][2] + new["ux"][3],
                         torch.where(vert, new["uz"][0] + new["uz"][2] + new["uz"][3], un))
        qn = 2 * q - Q[1] + dt ** 2 * V ** 2 * 2 * (E - D) * s2
        qn = torch.where(side, new["qx"][0] + new["qx"][2], qn)
        U, Q = [un, u], [qn, q]
        for a in F:
            F[a] = [new[a], F[a][0]]
        iit = it - half
        if iit > 1 or (iit == 1 and not low):
            rec[:, :, iit - 1] = un[:, rr - 1, nxl:nxl + rng]
    return rec


def exact(case, seed):
    kind = case["kind"]
    if kind == "elastic" and not case["free"]:
        return None  # the smoothing chain of the absorbing mode takes minutes
    k = _inputs(case, seed)
    with torch.no_grad():
        return {"acoustic": _exact_acoustic, "acoustic3d": _exact_acoustic, "gradient": _exact_gradient,
                "gradient3d": _exact_gradient, "visco": _exact_visco, "visco_gradient": _exact_visco_gradient,
                "viscoel": _exact_viscoel, "elastic": _exact_elastic, "vti": _exact_vti}[kind](case, k)

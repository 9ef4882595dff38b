"""The work a user of this package has it do, as measurable cases.

Every case goes through the public entry points of the package: the single-step
operators (forward and gradient), the persistent multi-shot plans (forward
traces, misfit and gradients), and the one-call helper that builds its plan for
the call.  A case is a dict of plain values; `prepare` makes what a program has
in hand before the call, `run` makes one pass, `work` counts what a pass cannot
do without, and `exact` computes the same outputs in 64 bits with torch alone.

Kinds:
  ac_op    acoustic_one_step and acoustic_one_step_grad (the drop-in operator)
  el_op    elastic_one_step and elastic_one_step_grad
  ac_fwd   AcousticPlan.forward: observed data of a survey
  ac_grad  AcousticPlan misfit and gradient: one FWI iteration
  ac_call  compute_loss_and_grads_GPU: the same with the plan made in the call
  el_fwd   ElasticPlan.forward
  el_grad  ElasticPlan misfit and gradients w.r.t. lambda, mu, rho

FP32 plans are run as a program with an FP32 model runs them: the model is an
FP32 tensor and the loss and gradients are kept in FP32 (the plans return them
in FP64 containers).
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

F64, F32 = torch.float64, torch.float32
VMIN, VMAX = 1500.0, 4500.0


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ------------------------------------------------------------------ the cases

def _case(kind, prec="f32", variant=0, nshots=1, nx=100, ny=100, nstep=1, npml=20, hx=10.0,
          hy=10.0, nrcv=0, resident=0, uneven=False, srcgrad=False, name=None):
    c = dict(kind=kind, prec=prec, variant=variant, nshots=nshots, nx=nx, ny=ny, nstep=nstep,
             npml=npml, hx=hx, hy=hy, nrcv=nrcv, resident=resident, uneven=uneven,
             srcgrad=srcgrad)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one call of the drop-in operator and its gradient at the smallest size the
        # reference's own forward benchmark sweeps (its default one_step form)
        _case("ac_op", "f64", 1, nx=101, ny=101, npml=12, name="ac_op_101_f64_u"),
        # the same operator pair at the top of that sweep, in the custom operators' form
        _case("ac_op", "f64", 0, nx=1001, ny=1001, npml=12, name="ac_op_1001_f64_w"),
        # one elastic step and its transpose on the elastic benchmark grid
        _case("el_op", "f64", nx=600, ny=300, npml=30, name="el_op_600_f64"),
        # observed data of one shot, plain FP64: the acoustic forward configuration
        _case("ac_fwd", "f64", 0, 1, 240, 240, 1000, 20, nrcv=200, name="ac_fwd_240_f64"),
        # FP64 FWI iteration of 8 shots on 400 x 400 (a quarter of that configuration's steps)
        _case("ac_grad", "f64", 0, 8, 400, 400, 500, 30, nrcv=340, name="ac_grad_400_f64"),
        # the batched FP32 FWI iteration (half the benchmark's shots, a fifth of its steps);
        # as there, about half of the checkpoint segments stay resident
        _case("ac_grad", "f32", 0, 32, 1000, 500, 600, 40, nrcv=500, resident=3,
              name="ac_grad_1000_f32"),
        # uneven apertures and record lengths on a 2000-cell-deep model, FP32
        _case("ac_grad", "f32", 0, 10, 1200, 2000, 400, 40, nrcv=300, uneven=True,
              name="ac_grad_uneven_f32"),
        # one small odd-sized shot in the reference's default one_step form, FP32
        _case("ac_grad", "f32", 1, 1, 187, 143, 500, 12, hy=8.0, nrcv=90,
              name="ac_grad_187_f32_u"),
        # the one-call gradient of the Marmousi example's size, its defaults (FP64, one_step);
        # the plan is made inside the call
        _case("ac_call", "f64", 1, 8, 200, 66, 800, 12, nrcv=183, name="ac_call_200_f64_u"),
        # elastic FWI iteration, FP32 (half the configuration's shots, a tenth of its steps)
        _case("el_grad", "f32", 0, 16, 600, 300, 400, 30, nrcv=300, resident=2,
              name="el_grad_600_f32"),
        # elastic FWI iteration in plain FP64 on a modest odd-sized grid
        _case("el_grad", "f64", 0, 2, 253, 187, 250, 12, nrcv=100, name="el_grad_253_f64"),
        # elastic observed data of one shot, FP32
        _case("el_fwd", "f32", 0, 1, 401, 201, 600, 20, nrcv=150, name="el_fwd_401_f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ac_op", "el_op", "ac_fwd", "ac_grad", "ac_grad", "ac_call", "el_fwd",
                       "el_grad", "el_grad"])
    prec = rng.choice(["f64", "f32"])
    variant = rng.choice([0, 1]) if kind.startswith("ac") else 0
    hx, hy = rng.choice([(10.0, 10.0), (10.0, 10.0), (12.5, 10.0), (20.0, 12.0)])
    npml = rng.choice([12, 20, 30, 40])
    if kind == "ac_op":
        return _case(kind, prec, variant, nx=_log(rng, 60, 1200), ny=_log(rng, 60, 1200),
                     npml=npml if npml < 30 else 12, hx=hx, hy=hy)
    if kind == "el_op":
        return _case(kind, prec, nx=_log(rng, 60, 700), ny=_log(rng, 60, 400), npml=12, hx=hx,
                     hy=hy)
    nx, ny = _log(rng, 110, 1100), _log(rng, 100, 600)
    if kind == "ac_call":
        nx, ny = _log(rng, 110, 400), _log(rng, 64, 200)
        npml = 12
    if kind.startswith("el"):
        nx, ny = _log(rng, 110, 620), _log(rng, 90, 320)
    nshots = 1 if kind.endswith("fwd") else _log(rng, 1, 24)
    nstep = rng.randint(150, 700)
    # at most about a quarter of the largest listed case of its kind
    most = {"ac_fwd": 1.2e8, "ac_grad": 2.4e9, "ac_call": 1.0e8, "el_fwd": 6e7,
            "el_grad": 2.4e8}[kind]
    if prec == "f64":
        most = min(most, 6e8 if kind.startswith("ac") else 4e7)
    nshots = int(max(1, min(nshots, most / (nx * ny * nstep))))
    nstep = int(max(60, min(nstep, most / (nx * ny * nshots))))
    npml = min(npml, (min(nx, ny) - 30) // 2)
    return _case(kind, prec, variant, nshots, nx, ny, nstep, npml, hx=hx, hy=hy,
                 nrcv=max(1, min(nx, 700) - 2 * npml - 3 - rng.randint(0, 20)),
                 resident=rng.choice([0, 0, -1, 2]) if kind.endswith("grad") else 0,
                 uneven=kind == "ac_grad" and rng.random() < 0.3,
                 # source inversion: the wavelet's gradient too
                 srcgrad=kind == "ac_grad" and prec == "f64" and rng.random() < 0.4)


# ------------------------------------------------------------------ inputs (torch, numpy only)

def _rand(seed, n, salt=0):
    g = torch.Generator().manual_seed(int(seed) * 1009 + salt)
    return torch.rand(n, generator=g, dtype=F64).tolist()


def _dt(c):
    """A step within the schemes' stability limits at the fastest model velocity."""
    s = math.sqrt(1 / c["hx"] ** 2 + 1 / c["hy"] ** 2)
    return (0.62 if c["kind"].startswith("ac") else 0.5) / (1.08 * VMAX * s)


def _velocity(c, seed, width):
    """A folded layered model with smooth anomalies, (width+2, ny+2) FP64."""
    r = _rand(seed, 64)
    d = _dev()
    x = torch.linspace(0, 1, width + 2, dtype=F64, device=d)[:, None]
    z = torch.linspace(0, 1, c["ny"] + 2, dtype=F64, device=d)[None, :]
    fold = 0.03 * torch.cos(2 * math.pi * (1 + 3 * r[0]) * x + 6 * r[1])
    n = 5
    v = torch.full((width + 2, c["ny"] + 2), VMIN, dtype=F64, device=d)
    for k in range(n):
        depth = (k + 0.5 + 0.6 * (r[2 + k] - 0.5)) / n
        v = v + (VMAX - VMIN) / n * torch.sigmoid((z + fold - depth) * 60)
    for k in range(4):
        a, b = r[20 + 2 * k], 0.2 + 0.7 * r[21 + 2 * k]
        v = v * (1 + 0.06 * (r[30 + k] - 0.5) * torch.exp(-((x - a) ** 2 + (z - b) ** 2) / 0.01))
    return v


def _ricker(nstep, dt, f):
    t = np.arange(nstep) * dt - 1.2 / f
    a = (math.pi * f * t) ** 2
    return (1 - 2 * a) * np.exp(-a)


def _shots(c, seed):
    """The survey: per shot its window, record length, source and receivers (1-based)."""
    out = []
    r = _rand(seed, 3 * c["nshots"] + 3, salt=1)
    dt, npml = _dt(c), c["npml"]
    for s in range(c["nshots"]):
        nx, nstep, x0 = c["nx"], c["nstep"], 0
        if c["uneven"]:  # apertures and record lengths of a third to all of the largest
            f = (s + 0.5) / c["nshots"]
            nx = max(2 * npml + 30, int(c["nx"] * (1 / 3 + 2 / 3 * ((f * 5) % 1))))
            nstep = max(40, int(c["nstep"] * (1 / 3 + 2 / 3 * ((f * 3 + 0.3) % 1))))
            x0 = int(r[3 * s + 1] * (_model_width(c) - nx))
        pos = (s + 0.5) / c["nshots"] if not c["uneven"] else 0.3 + 0.4 * r[3 * s]
        si = npml + 4 + int(pos * (nx - 2 * npml - 6))
        n = max(1, min(c["nrcv"], nx - 2 * npml - 2))
        rcvi = np.round(np.linspace(npml + 2, nx - npml, n)).astype(np.int64)
        amp = 1e6 * (0.8 + 0.4 * r[3 * s + 2])
        out.append(dict(x0=x0, nx=nx, nstep=nstep, si=si, sj=npml + 8, rcvi=rcvi, rj=npml + 5,
                        wav=amp * _ricker(nstep, dt, 0.06 * VMIN / max(c["hx"], c["hy"]))))
    return out


def _model_width(c):
    return 3 * c["nx"] if c["uneven"] else c["nx"]


def _observed(c, s, seed, k, scale):
    """(nstep+1, nrcv) field records of shot k: a direct and a reflected arrival
    with the shot's wavelet."""
    d, dt = _dev(), _dt(c)
    r = _rand(seed, 4, salt=50 + k)
    t = torch.arange(s["nstep"] + 1, dtype=F64, device=d)[:, None] * dt
    x = (torch.as_tensor(s["rcvi"], device=d).to(F64) - s["si"])[None, :] * c["hx"]
    f = 0.06 * VMIN / max(c["hx"], c["hy"])
    rec = torch.zeros(s["nstep"] + 1, len(s["rcvi"]), dtype=F64, device=d)
    for depth, a in ((3 * c["hy"], 1.0), ((0.2 + 0.3 * r[0]) * c["ny"] * c["hy"], 0.3)):
        dist = torch.sqrt(x * x + 4 * depth * depth)
        q = (math.pi * f * (t - 1.2 / f - dist / (VMIN * (1 + 0.3 * r[1])))) ** 2
        rec = rec + a * (1 - 2 * q) * torch.exp(-q) / torch.sqrt(1 + dist / (20 * c["hx"]))
    return scale * rec


def _elastic_model(c, seed):
    """(lambda, mu, rho) on the (nx+2, ny+2) grid, FP64."""
    vp = _velocity(c, seed, c["nx"])
    vs = vp / math.sqrt(3.0)
    rho = 310.0 * vp ** 0.25
    mu = rho * vs * vs
    return rho * vp * vp - 2 * mu, mu, rho


def _typed(c, x):
    return x.to(F64 if c["prec"] == "f64" else F32)


# amplitude of the acoustic and elastic field records (the traces' own scale)
AC_OBS, EL_OBS = 2.0, 0.05


# ------------------------------------------------------------------ prepare and run

def _op_inputs(c, seed):
    """Fields of a running simulation: smooth wave packets, the model, the PML."""
    d = _dev()
    n = (c["nx"] + 2) * (c["ny"] + 2)
    x = torch.arange(c["nx"] + 2, dtype=F64, device=d)[:, None]
    z = torch.arange(c["ny"] + 2, dtype=F64, device=d)[None, :]
    r = _rand(seed, 200, salt=3)
    it = iter(r)

    def field(scale=1.0):
        a, b, p, w = (next(it) for _ in range(4))
        g = torch.sin(0.25 * (0.4 + a) * x + 6 * p) * torch.cos(0.25 * (0.4 + b) * z + 5 * w)
        g = scale * g * torch.exp(-((x / c["nx"] - a) ** 2 + (z / c["ny"] - b) ** 2) * 3)
        g[0], g[-1], g[:, 0], g[:, -1] = 0, 0, 0, 0
        return g.reshape(n)

    return field


def prepare(case, seed):
    ads = load_package()
    c = case
    kind = c["kind"]
    st = dict(case=c, ads=ads)
    dt = _dt(c)
    if kind == "ac_op":
        f = _op_inputs(c, seed)
        s, t = _pml_2d(c)
        vp = _velocity(c, seed, c["nx"]).reshape(-1)
        st["ins"] = [_typed(c, v) for v in (f(), f(), f(10.0), f(10.0), s, t, vp * vp)]
        st["gs"] = [_typed(c, f()) for _ in range(3)]
        st["k"] = (dt, c["hx"], c["hy"], c["nx"], c["ny"])
        return st
    if kind == "el_op":
        f = _op_inputs(c, seed)
        st["param"] = ads.ElasticPropagatorParams(
            NX=c["nx"], NY=c["ny"], NSTEP=1, DELTAX=c["hx"], DELTAY=c["hy"], DELTAT=dt,
            NPOINTS_PML=c["npml"], vp_ref=3000.0, f0=10.0)
        st["model"] = [_typed(c, v.reshape(-1)) for v in _elastic_model(c, seed)]
        st["state"], st["gout"] = (_typed(c, v) for v in _el_op_fields(f, c))
        st["prof"] = [_typed(c, torch.as_tensor(p, device=_dev())) for p in _cpml(c)]
        st["src"] = _el_op_source(c)
        return st
    shots = _shots(c, seed)
    if kind.startswith("ac"):
        vp = _velocity(c, seed, _model_width(c))
        st["vp"] = _typed(c, vp)
        obs = [_observed(c, s, seed, k, AC_OBS) for k, s in enumerate(shots)]
        if kind == "ac_call":
            st["param"] = ads.AcousticPropagatorParams(
                NX=c["nx"], NY=c["ny"], NSTEP=c["nstep"], DELTAX=c["hx"], DELTAY=c["hy"],
                DELTAT=dt, NPOINTS_PML=c["npml"], vp_ref=1000.0,
                PropagatorKernel=0 if c["variant"] else 1)
            st["srcs"] = [ads.AcousticSource(np.array([s["si"]]), np.array([s["sj"]]),
                                             s["wav"][:, None]) for s in shots]
            st["rcvs"] = [ads.AcousticReceiver(s["rcvi"], np.full(len(s["rcvi"]), s["rj"]))
                          for s in shots]
            st["Rs"] = [_typed(c, o) for o in obs]
            return st
        st["plan"] = ads.AcousticPlan(
            _model_width(c), c["ny"], c["hx"], c["hy"], dt,
            [dict(x0=s["x0"], nx=s["nx"], nstep=s["nstep"], srci=[s["si"]], srcj=[s["sj"]],
                  srcv=s["wav"][:, None], rcvi=s["rcvi"],
                  rcvj=np.full(len(s["rcvi"]), s["rj"])) for s in shots],
            npml=c["npml"], vp_ref=1000.0, precision=c["prec"], variant=c["variant"],
            resident_segments=c["resident"])
        st["obs"] = _typed(c, torch.cat([o.reshape(-1) for o in obs]))
        return st
    st["model"] = [_typed(c, v) for v in _elastic_model(c, seed)]
    p = ads.ElasticPropagatorParams(NX=c["nx"], NY=c["ny"], NSTEP=c["nstep"], DELTAX=c["hx"],
                                    DELTAY=c["hy"], DELTAT=dt, NPOINTS_PML=c["npml"],
                                    vp_ref=3000.0, f0=10.0)
    st["plan"] = ads.ElasticPlan(
        p, [dict(srci=[s["si"]] * 2, srcj=[s["sj"]] * 2, srctype=[2, 3],
                 srcv=np.repeat(s["wav"][:, None], 2, axis=1),
                 rcvi=np.concatenate([s["rcvi"], s["rcvi"]]),
                 rcvj=np.full(2 * len(s["rcvi"]), s["rj"]),
                 rcvtype=np.repeat([0, 1], len(s["rcvi"]))) for s in shots],
        precision=c["prec"], resident_segments=c["resident"])
    # records are (nrcv, nstep+1): x then y components
    st["obs"] = _typed(c, torch.cat([_el_observed(c, s, seed, k).reshape(-1)
                                     for k, s in enumerate(shots)]))
    return st


def _el_observed(c, s, seed, k):
    o = _observed(c, s, seed, k, EL_OBS).T
    return torch.cat([o, 0.7 * o])


def _el_op_fields(f, c):
    """Velocities of order 1e-2 and stresses of order 1e5, as the plans' shots have them."""
    scale = [1e-2, 1e-2, 1e5, 1e5, 1e5] + [1e-4] * 4 + [1e3] * 4
    return (torch.stack([f(a) for a in scale]),
            torch.stack([f(1.0 / a) for a in scale]))


def _el_op_source(c):
    return dict(srci=[c["nx"] // 2] * 2, srcj=[c["npml"] + 8] * 2, srctype=[2, 3],
                srcv=np.array([3e4, 3e4]))


def run(state):
    c, ads = state["case"], state["ads"]
    kind = c["kind"]
    if kind == "ac_op":
        out = ads.acoustic_one_step(*state["ins"], *state["k"], c["variant"])
        grads = ads.acoustic_one_step_grad(*state["gs"], *state["ins"], *state["k"], *out,
                                           c["variant"])
        return list(out) + list(grads)
    if kind == "el_op":
        lam, mu, rho = state["model"]
        new = ads.elastic_one_step(state["param"], rho, lam, mu, state["state"], state["prof"],
                                   **state["src"])
        return [new] + list(ads.elastic_one_step_grad(state["param"], rho, lam, mu,
                                                      state["state"], state["gout"],
                                                      state["prof"]))
    if kind == "ac_call":
        out = ads.compute_loss_and_grads_GPU(state["param"], state["srcs"], state["rcvs"],
                                             state["Rs"], state["vp"], precision=c["prec"])
        return [_typed(c, v) for v in out]
    plan = state["plan"]
    if kind == "ac_fwd":
        return [plan.forward(state["vp"])]
    if kind == "ac_grad":
        loss, grad, *more = plan.gradient(state["vp"], state["obs"],
                                          want_source_grad=c["srcgrad"])
        return [_typed(c, v) for v in [loss, grad] + [g for m in more for g in m]]
    if kind == "el_fwd":
        return [plan.forward(*state["model"])]
    return [_typed(c, v) for v in plan.gradient(*state["model"], state["obs"])]


# ------------------------------------------------------------------ work

def work(case):
    """Inputs and outputs once each, and the arithmetic of one step of the scheme
    per cell and time step (multiplications and additions of the wave update
    outside the absorbing layers)."""
    c = case
    b = 8 if c["prec"] == "f64" else 4
    n = (c["nx"] + 2) * (c["ny"] + 2)
    if c["kind"] == "ac_op":
        return dict(bytes=b * n * (7 + 3 + 3 + 5), flops=n * (30 + 60))
    if c["kind"] == "el_op":
        return dict(bytes=b * n * (3 + 13 + 13 + 13 + 13 + 3), flops=n * (110 + 170))
    shots = _shots(c, 0)
    steps = sum(s["nx"] * c["ny"] * s["nstep"] for s in shots)
    traces = sum((s["nstep"] + 1) * len(s["rcvi"]) for s in shots)
    m = (_model_width(c) + 2) * (c["ny"] + 2)
    if c["kind"] == "ac_fwd":
        return dict(bytes=b * (m + traces), flops=steps * 9)
    if c["kind"] in ("ac_grad", "ac_call"):
        return dict(bytes=b * (2 * m + traces), flops=steps * (9 + 18))
    if c["kind"] == "el_fwd":
        return dict(bytes=b * (3 * m + 2 * traces), flops=steps * 60)
    return dict(bytes=b * (6 * m + 2 * traces), flops=steps * (60 + 90))


# ------------------------------------------------------------------ 64-bit values, torch only

def _profile(n, h, npml, v):
    """Damping of the acoustic PML along one axis (padded indices 0..n+1)."""
    L = npml * h
    xi = v / L * math.log(1 / 0.001)
    x = np.arange(n + 2) * h
    far = h * (n + 1) - L
    d = np.where(x < L, np.abs(L - x), np.where(x > far, np.abs(x - far), 0.0))
    return xi * (d / L - np.sin(2 * math.pi * d / L) / (2 * math.pi))


def _pml_1d(c, nx):
    d = _dev()
    return (torch.as_tensor(_profile(nx, c["hx"], c["npml"], 1000.0), device=d)[:, None],
            torch.as_tensor(_profile(c["ny"], c["hy"], c["npml"], 1000.0), device=d)[None, :])


def _pml_2d(c):
    s, t = _pml_1d(c, c["nx"])
    shape = (c["nx"] + 2, c["ny"] + 2)
    return s.expand(shape).reshape(-1).contiguous(), t.expand(shape).reshape(-1).contiguous()


def _cpml(c):
    """(ax, bx, kx, ay, by, ky) of the elastic step: (2, n), integer and half grid."""
    dt, out = _dt(c), []
    alpha_max = math.pi * 10.0
    for n, h in ((c["nx"], c["hx"]), (c["ny"], c["hy"])):
        thick = c["npml"] * h
        d0 = -3.0 * 3000.0 * math.log(0.001) / (2 * thick)
        pos = h * np.arange(n)[None, :] + np.array([[0.0], [h / 2]])
        lo, hi = (thick - pos) / thick, (pos - ((n - 0.5) * h - thick)) / thick
        u = np.where(hi >= 0, hi, np.where(lo >= 0, lo, 0.0))
        d, al = d0 * u ** 2, np.where((hi >= 0) | (lo >= 0), alpha_max * u, 0.0)
        bb = np.exp(-(d + al) * dt)
        with np.errstate(invalid="ignore", divide="ignore"):
            aa = np.where(np.abs(d) > 1e-6, d * (bb - 1) / (d + al), 0.0)
        out += [aa, bb, np.ones_like(bb)]
    return out


def _pad(x):
    return torch.nn.functional.pad(x, (1, 1, 1, 1))


def _ac_step(w, wo, p, q, s, t, cc, dt, hx, hy, variant):
    """One acoustic step on (..., nx+2, ny+2) FP64 fields (s, t broadcast or full)."""
    I = (Ellipsis, slice(1, -1), slice(1, -1))
    N, S = (Ellipsis, slice(2, None), slice(1, -1)), (Ellipsis, slice(None, -2), slice(1, -1))
    R, L = (Ellipsis, slice(1, -1), slice(2, None)), (Ellipsis, slice(1, -1), slice(None, -2))
    sg, ta = (v[1:-1] if v.shape[0] > 1 else v for v in (s, t))
    sg, ta = (v[:, 1:-1] if v.shape[1] > 1 else v for v in (sg, ta))
    C = cc[I]
    cx, cy = (dt / hx) ** 2, (dt / hy) ** 2
    W = w[I]
    u = ((2 - sg * ta * dt * dt - 2 * (cx + cy) * C) * W + C * (cx * (w[N] + w[S]) +
         cy * (w[R] + w[L])) + dt * dt / (2 * hx) * (p[N] - p[S]) +
         dt * dt / (2 * hy) * (q[R] - q[L]) - (1 - (sg + ta) * dt / 2) * wo[I])
    u = _pad(u / (1 + (sg + ta) / 2 * dt))
    f = u if variant else w
    p2 = (1 - dt * sg) * p[I] + dt / (2 * hx) * C * (ta - sg) * (f[N] - f[S])
    q2 = (1 - dt * ta) * q[I] + dt / (2 * hy) * C * (sg - ta) * (f[R] - f[L])
    return u, _pad(p2), _pad(q2)


def _box(f, b, di=0, dj=0):
    i0, i1, j0, j1 = b
    return f[..., i0 + di:i1 + 1 + di, j0 + dj:j1 + 1 + dj]


def _el_step(F, model, prof, dt, hx, hy):
    """One elastic step: F the 13 fields, (..., nx+2, ny+2) FP64 each."""
    vx, vy, sxx, syy, sxy = F[:5]
    m = F[5:]
    lam, mu, rho = model
    nx, ny = lam.shape[0] - 2, lam.shape[1] - 2
    (axi, axh), (bxi, bxh), (ayi, ayh), (byi, byh) = prof
    X = lambda v, b: v[b[0] - 1:b[1], None]
    Y = lambda v, b: v[None, b[2] - 1:b[3]]

    def d(f, b, axis, fwd, h):  # staggered difference, forward or backward
        k = (1, 0, 2, -1) if fwd else (0, -1, 1, -2)
        g = [_box(f, b, a, 0) if axis == 0 else _box(f, b, 0, a) for a in k]
        return (27 * (g[0] - g[1]) - g[2] + g[3]) / (24 * h)

    def put(x, b):  # a box's values on the padded grid
        return torch.nn.functional.pad(x, (b[2], ny + 1 - b[3], b[0], nx + 1 - b[1]))

    b1, b2 = (1, nx - 1, 2, ny), (2, nx, 1, ny - 1)
    b3, b4 = (2, nx, 2, ny), (1, nx - 1, 1, ny - 1)
    dvx, dvy = d(vx, b1, 0, True, hx), d(vy, b1, 1, False, hy)
    m1 = X(bxh, b1) * _box(m[0], b1) + X(axh, b1) * dvx
    m2 = Y(byi, b1) * _box(m[1], b1) + Y(ayi, b1) * dvy
    la = (_box(lam, b1, 1) + _box(lam, b1)) / 2
    lm = la + _box(mu, b1, 1) + _box(mu, b1)
    e1, e2 = dvx + m1, dvy + m2
    sxx = sxx + put(dt * (lm * e1 + la * e2), b1)
    syy = syy + put(dt * (lm * e2 + la * e1), b1)
    dyx, dxy = d(vy, b2, 0, False, hx), d(vx, b2, 1, True, hy)
    m3 = X(bxi, b2) * _box(m[2], b2) + X(axi, b2) * dyx
    m4 = Y(byh, b2) * _box(m[3], b2) + Y(ayh, b2) * dxy
    sxy = sxy + put(dt * (_box(mu, b2) + _box(mu, b2, 0, 1)) / 2 * (dyx + m3 + dxy + m4), b2)
    a, b = d(sxx, b3, 0, False, hx), d(sxy, b3, 1, False, hy)
    m5 = X(bxi, b3) * _box(m[4], b3) + X(axi, b3) * a
    m6 = Y(byi, b3) * _box(m[5], b3) + Y(ayi, b3) * b
    vx = vx + put((a + m5 + b + m6) * dt / _box(rho, b3), b3)
    a, b = d(sxy, b4, 0, True, hx), d(syy, b4, 1, True, hy)
    m7 = X(bxh, b4) * _box(m[6], b4) + X(axh, b4) * a
    m8 = Y(byh, b4) * _box(m[7], b4) + Y(ayh, b4) * b
    r4 = (_box(rho, b4) + _box(rho, b4, 1) + _box(rho, b4, 1, 1) + _box(rho, b4, 0, 1)) / 4
    vy = vy + put((a + m7 + b + m8) * dt / r4, b4)
    return [vx, vy, sxx, syy, sxy, put(m1, b1), put(m2, b1), put(m3, b2), put(m4, b2),
            put(m5, b3), put(m6, b3), put(m7, b4), put(m8, b4)]


def _sweep(state, step, first, nstep, obs_of, params, want_grad, seg):
    """Time loop `state, rec = step(n, state)` for n = first..nstep, and the gradient of
    sum (rec_n - obs_n)^2 w.r.t. `params` by recomputing segments of `seg` steps under
    autograd.  Returns (records, loss, gradients)."""
    marks, recs = [], []
    with torch.no_grad():
        for n in range(first, nstep + 1):
            if (n - first) % seg == 0:
                marks.append((n, [v.clone() for v in state]))
            state, rec = step(n, state)
            recs.append(rec)
    if not want_grad:
        return recs, None, None
    loss = sum(torch.sum((r - obs_of(first + k)) ** 2) for k, r in enumerate(recs))
    lam = [torch.zeros_like(v) for v in state]
    grads = [torch.zeros_like(p) for p in params]
    for n0, s0 in reversed(marks):
        ins = [v.requires_grad_(True) for v in s0]
        s, part = ins, 0.0
        for n in range(n0, min(n0 + seg, nstep + 1)):
            s, rec = step(n, s)
            part = part + torch.sum((rec - obs_of(n)) ** 2)
        part = part + sum(torch.sum(a * b) for a, b in zip(lam, s))
        got = torch.autograd.grad(part, ins + params, allow_unused=True)
        lam = [torch.zeros_like(v) if g is None else g for g, v in zip(got, ins)]
        grads = [a if g is None else a + g for a, g in zip(grads, got[len(ins):])]
        del s, part, got, ins
    return recs, loss, grads


def _seg(cells, fields):
    return int(max(2, min(64, 30e9 / (8.0 * cells * fields))))


def _groups(c, shots):
    """Shots computed together: equal windows and record lengths, about 4M cells."""
    if c["uneven"]:
        return [[k] for k in range(len(shots))]
    n = max(1, int(4e6 / ((c["nx"] + 2) * (c["ny"] + 2))))
    return [list(range(a, min(a + n, len(shots)))) for a in range(0, len(shots), n)]


def _exact_acoustic(c, seed, grad):
    d, dt = _dev(), _dt(c)
    shots = _shots(c, seed)
    vp_all = _typed(c, _velocity(c, seed, _model_width(c))).to(F64)
    gvp = torch.zeros_like(vp_all)
    loss, traces, gsrc = 0.0, [None] * len(shots), [None] * len(shots)
    for group in _groups(c, shots):
        g0 = shots[group[0]]
        nx, nstep, B = g0["nx"], g0["nstep"], len(group)
        s, t = _pml_1d(c, nx)
        vp = vp_all[g0["x0"]:g0["x0"] + nx + 2].clone().requires_grad_(grad)
        src = torch.as_tensor(np.stack([shots[k]["wav"] for k in group]), device=d)
        src = src.clone().requires_grad_(grad)
        bi = torch.arange(B, device=d)
        si = torch.tensor([shots[k]["si"] - 1 for k in group], device=d)
        sj = torch.tensor([shots[k]["sj"] - 1 for k in group], device=d)
        ri = torch.stack([torch.as_tensor(shots[k]["rcvi"] - 1, device=d) for k in group])
        rj = g0["rj"] - 1
        obs = torch.stack([_typed(c, _observed(c, shots[k], seed, k, AC_OBS)).to(F64)
                           for k in group])

        def step(n, S):
            u, p, q = _ac_step(*S, s, t, vp * vp, dt, c["hx"], c["hy"], c["variant"])
            u = u.index_put((bi, si, sj), src[:, n - 1] * dt * dt, accumulate=True)
            return [u, S[0], p, q], u[bi[:, None], ri, rj]

        z = torch.zeros(B, nx + 2, c["ny"] + 2, dtype=F64, device=d)
        recs, l, gr = _sweep([z, z, z, z], step, 2, nstep, lambda n: obs[:, n], [vp, src], grad,
                             _seg(z.numel(), 40))
        zero = torch.zeros_like(recs[0])
        tr = torch.stack([zero, zero] + recs, dim=1)
        for b, k in enumerate(group):
            traces[k] = tr[b]
        if grad:
            loss = loss + l + torch.sum(obs[:, :2] ** 2)
            gvp[g0["x0"]:g0["x0"] + nx + 2] += gr[0]
            for b, k in enumerate(group):
                gsrc[k] = gr[1][b][:, None]
    if not grad:
        return [torch.cat([v.reshape(-1) for v in traces])]
    return [loss, gvp] + (gsrc if c["srcgrad"] else [])


def _exact_elastic(c, seed, grad):
    d, dt = _dev(), _dt(c)
    shots = _shots(c, seed)
    model = [_typed(c, v).to(F64).clone().requires_grad_(grad) for v in _elastic_model(c, seed)]
    P = [torch.as_tensor(p, device=d) for p in _cpml(c)]
    prof = (P[0], P[1], P[3], P[4])
    loss, traces = 0.0, [None] * len(shots)
    total = [torch.zeros_like(v) for v in model]
    for group in _groups(c, shots):
        g0, B = shots[group[0]], len(group)
        src = torch.as_tensor(np.stack([shots[k]["wav"] for k in group]), device=d)
        bi = torch.arange(B, device=d)
        si = torch.tensor([shots[k]["si"] - 1 for k in group], device=d)
        sj = torch.tensor([shots[k]["sj"] - 1 for k in group], device=d)
        ri = torch.stack([torch.as_tensor(shots[k]["rcvi"] - 1, device=d) for k in group])
        rj = g0["rj"] - 1
        obs = torch.stack([_typed(c, _el_observed(c, shots[k], seed, k)).to(F64) for k in group])

        def step(n, S):
            S = _el_step(S, model, prof, dt, c["hx"], c["hy"])
            for f in (2, 3):
                S[f] = S[f].index_put((bi, si, sj), src[:, n - 1], accumulate=True)
            return S, torch.cat([S[f][bi[:, None], ri, rj] for f in (0, 1)], dim=1)

        z = torch.zeros(B, c["nx"] + 2, c["ny"] + 2, dtype=F64, device=d)
        recs, l, gr = _sweep([z] * 13, step, 1, g0["nstep"], lambda n: obs[:, :, n], model, grad,
                             _seg(z.numel(), 160))
        tr = torch.stack([torch.zeros_like(recs[0])] + recs, dim=2)
        for b, k in enumerate(group):
            traces[k] = tr[b]
        if grad:
            loss = loss + l + torch.sum(obs[:, :, 0] ** 2)
            total = [a + b for a, b in zip(total, gr)]
    if not grad:
        return [torch.cat([v.reshape(-1) for v in traces])]
    return [loss] + total


def _exact_op(c, seed):
    dt = _dt(c)
    f = _op_inputs(c, seed)
    shape = (c["nx"] + 2, c["ny"] + 2)
    if c["kind"] == "ac_op":
        s, t = (_typed(c, v).to(F64).view(shape) for v in _pml_2d(c))
        vp = _velocity(c, seed, c["nx"])
        ins = [_typed(c, f(a)).to(F64).view(shape).requires_grad_(True) for a in (1, 1, 10.0, 10.0)]
        cc = _typed(c, vp * vp).to(F64).requires_grad_(True)
        gs = [_typed(c, f()).to(F64).view(shape) for _ in range(3)]
        out = _ac_step(*ins, s, t, cc, dt, c["hx"], c["hy"], c["variant"])
        got = torch.autograd.grad(sum(torch.sum(a * b) for a, b in zip(out, gs)), ins + [cc])
        return [v.detach().reshape(-1) for v in list(out) + list(got)]
    state, gout = (_typed(c, v).to(F64).view(13, *shape) for v in _el_op_fields(f, c))
    model = [_typed(c, v).to(F64).requires_grad_(True) for v in _elastic_model(c, seed)]
    P = [_typed(c, torch.as_tensor(p, device=_dev())).to(F64) for p in _cpml(c)]
    ins = [v.clone().requires_grad_(True) for v in state]
    out = _el_step(ins, model, (P[0], P[1], P[3], P[4]), dt, c["hx"], c["hy"])
    got = torch.autograd.grad(sum(torch.sum(a * b) for a, b in zip(out, gout)), ins + model)
    src, new = _el_op_source(c), torch.stack(out).detach()
    for i, j, k, v in zip(src["srci"], src["srcj"], src["srctype"], src["srcv"]):
        new[k, i - 1, j - 1] += v
    n = shape[0] * shape[1]
    return [new.reshape(13, n), torch.stack(got[:13]).reshape(13, n)] + [g.reshape(-1)
                                                                         for g in got[13:]]


def exact(case, seed):
    c = case
    if c["kind"].endswith("op"):
        return _exact_op(c, seed)
    grad = not c["kind"].endswith("fwd")
    return (_exact_acoustic if c["kind"].startswith("ac") else _exact_elastic)(c, seed, grad)

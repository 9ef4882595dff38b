"""FP64 acoustic plans against extended precision.

The step's weights have to cancel on a constant field as well as FP64 allows: where the
centre weight is rounded apart from the others, every step carries the same small mass
term, and the error grows with the record instead of like a random walk.  The bound is
what the arithmetic allows: four times the error of a plain FP64 numpy restatement in
difference form, whose weights cancel exactly."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def profile(n, h, npml, vref):
    L = npml * h
    x = np.arange(n + 2) * h
    far = h * (n + 1) - L
    d = np.where(x < L, np.abs(L - x), np.where(x > far, np.abs(x - far), 0.0))
    return vref / L * math.log(1000) * (d / L - np.sin(2 * math.pi * d / L) / (2 * math.pi))


def restated(T, nx, ny, nstep, hx, hy, dt, sg, ta, vp, wav, si, sj, rows, rj):
    """Traces of the w form in difference form, all arithmetic in type T."""
    dt, hx, hy = T(dt), T(hx), T(hy)
    sg, ta = sg.astype(T)[1:-1, None], ta.astype(T)[None, 1:-1]
    c = (vp.astype(T) ** 2)[1:-1, 1:-1]
    cx, cy, fx, fy = (dt / hx) ** 2, (dt / hy) ** 2, dt * dt / (2 * hx), dt * dt / (2 * hy)
    s = sg + ta
    w, wo, p, q = (np.zeros((nx + 2, ny + 2), T) for _ in range(4))
    out = np.zeros((nstep + 1, len(rows)), T)
    for t in range(2, nstep + 1):
        W, O, P, Q = (f[1:-1, 1:-1] for f in (w, wo, p, q))
        N, S, E, V = w[2:, 1:-1], w[:-2, 1:-1], w[1:-1, 2:], w[1:-1, :-2]
        d = ((1 - s * dt / 2) * (W - O) + c * (cx * ((N - W) + (S - W)) + cy * ((E - W) + (V - W)))
             - sg * ta * dt * dt * W + fx * (p[2:, 1:-1] - p[:-2, 1:-1])
             + fy * (q[1:-1, 2:] - q[1:-1, :-2])) / (1 + s * dt / 2)
        p2 = (1 - dt * sg) * P + dt / (2 * hx) * c * (ta - sg) * (N - S)
        q2 = (1 - dt * ta) * Q + dt / (2 * hy) * c * (sg - ta) * (E - V)
        new = np.zeros_like(w)
        new[1:-1, 1:-1] = W + d
        new[si, sj] += T(wav[t - 1]) * dt * dt
        p, q = np.zeros_like(p), np.zeros_like(q)
        p[1:-1, 1:-1], q[1:-1, 1:-1] = p2, q2
        wo, w = w, new
        out[t] = w[rows, rj]
    return out


@pytest.mark.parametrize("hx,hy", [(10.0, 10.0), (10.0, 8.0), (12.5, 10.0)])
def test_step_weights_cancel(ads, cuda, hx, hy):
    nx, ny, nstep, npml, vref = 84, 70, 500, 12, 1000.0
    dt = 0.62 / (1.08 * 4500 * math.sqrt(1 / hx ** 2 + 1 / hy ** 2))
    rng = np.random.default_rng(7)
    z = np.linspace(0, 1, ny + 2)[None, :]
    x = np.linspace(0, 1, nx + 2)[:, None]
    vp = 1500 + 3000 / (1 + np.exp(-12 * (z + 0.03 * np.cos(9 * x) - 0.5)))
    f = 90.0 / max(hx, hy)
    a = (np.pi * f * (np.arange(nstep) * dt - 1.2 / f)) ** 2
    wav = 1e6 * (1 - 2 * a) * np.exp(-a) * (1 + 1e-3 * rng.random(nstep))
    rows = np.arange(npml + 1, nx - npml)
    geo = (nx, ny, nstep, hx, hy, dt, profile(nx, hx, npml, vref), profile(ny, hy, npml, vref), vp,
           wav, nx // 2, npml + 7, rows, npml + 4)
    true = restated(np.longdouble, *geo)

    def err(r):
        return float(np.sqrt(((r.astype(np.longdouble) - true) ** 2).sum() / (true ** 2).sum()))

    shot = dict(x0=0, nx=nx, nstep=nstep, srci=[nx // 2 + 1], srcj=[npml + 8], srcv=wav[:, None],
                rcvi=rows + 1, rcvj=np.full(len(rows), npml + 5))
    plan = ads.AcousticPlan(nx, ny, hx, hy, dt, [shot], npml=npml, vp_ref=vref, precision="f64")
    got = plan.forward(torch.as_tensor(vp, dtype=torch.float64, device=cuda)).cpu().numpy()
    plan.close()
    assert err(got.reshape(nstep + 1, -1)) <= 4 * err(restated(np.float64, *geo))

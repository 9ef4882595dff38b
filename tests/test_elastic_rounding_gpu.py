"""The elastic stress update rounds a stress once a step, at its own size: from a state
whose stresses are 2^20 times the increments the velocities give them, the operator's new
stress is the sum rounded once, so it lies within half an ulp of the exact one (and the
increment's own rounding, some ulps of 2^-20 of it)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_operator_rounds_a_stress_once(ads, cuda, dtype):
    NX, NY = 61, 45
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=1, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=0.7e-3, NPOINTS_PML=1, vp_ref=3000.0, f0=15.0)
    rng = np.random.default_rng(3)
    T = np.float32 if dtype == torch.float32 else np.float64
    W = np.float64 if dtype == torch.float32 else np.longdouble
    shape = (NX + 2, NY + 2)
    lam, mu, rho = (np.full(shape, v) for v in (8e9, 6e9, 2200.0))
    st = np.zeros((13, *shape), T)
    st[0], st[1] = (rng.standard_normal(shape).astype(T) for _ in range(2))
    inc = 8e9 * 0.7e-3 * 27 / 24 / 8
    st[2:5] = inc * 2.0 ** 20 * (1 + rng.random((3, *shape)))
    # no absorbing layer: a = 0, b = 1
    prof = [np.zeros((2, NX)), np.ones((2, NX)), np.ones((2, NX)),
            np.zeros((2, NY)), np.ones((2, NY)), np.ones((2, NY))]
    t = lambda a: torch.as_tensor(a, dtype=dtype, device=cuda)
    out = ads.elastic_one_step(p, t(rho).reshape(-1), t(lam).reshape(-1), t(mu).reshape(-1),
                               t(st).reshape(13, -1), [t(a) for a in prof])
    out = out.cpu().numpy().reshape(13, *shape)
    vx, vy, sxx, syy = (a.astype(W) for a in st[:4])
    i, j = slice(4, NX - 3), slice(4, NY - 3)
    at = lambda f, a, b: f[4 + a:NX - 3 + a, 4 + b:NY - 3 + b]
    dt, hx, hy = W(p.DELTAT), W(10), W(8)
    e1 = (27 * (at(vx, 1, 0) - at(vx, 0, 0)) - at(vx, 2, 0) + at(vx, -1, 0)) / (24 * hx)
    e2 = (27 * (at(vy, 0, 0) - at(vy, 0, -1)) - at(vy, 0, 1) + at(vy, 0, -2)) / (24 * hy)
    for k, s, a, b in ((2, sxx, e1, e2), (3, syy, e2, e1)):
        exact = at(s, 0, 0) + dt * (W(20e9) * a + W(8e9) * b)
        ulp = np.spacing(np.abs(exact).astype(T)).astype(W)
        assert float((np.abs(out[k, i, j].astype(W) - exact) / ulp).max()) <= 0.5 + 1e-3

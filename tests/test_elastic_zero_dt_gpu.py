"""The transpose of an elastic step of no length: the state's gradient comes back as it
is, the memory variables' parts with it, and the parameters' gradients are zero."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_zero_dt(ads, orc, cuda, dtype):
    NX, NY = 40, 35
    N = (NX + 2) * (NY + 2)
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=1, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=0.7e-3, NPOINTS_PML=6, vp_ref=3000.0, f0=15.0)
    prof = ads.compute_elastic_PML_Params(p)
    p.DELTAT = 0.0
    rng = np.random.default_rng(2)
    f = lambda a: torch.as_tensor(np.asarray(a), dtype=dtype, device=cuda)
    lam, mu, rho = (1.0 + rng.random(N) for _ in range(3))
    st, w = rng.standard_normal((13, N)), rng.standard_normal((13, N))
    got = ads.elastic_one_step_grad(p, f(rho), f(lam), f(mu), f(st), f(w), [f(a) for a in prof])
    r = lambda a: f(a).double().cpu().numpy().reshape(-1)
    ax, bx, kx, ay, by, ky = (r(a) for a in prof)
    ref = orc.elastic_step_bwd(r(st), r(w), r(lam), r(mu), r(rho), ax, bx, ay, by, 0.0, 10.0, 8.0,
                               NX, NY)
    for a, b in zip(got, ref):
        a, b = a.double().cpu().numpy().reshape(-1), np.asarray(b).reshape(-1)
        assert np.linalg.norm(a - b) <= (1e-13 if dtype == torch.float64 else 1e-5) * max(
            np.linalg.norm(b), 1e-30)
    assert all(float(a.abs().max()) == 0.0 for a in got[1:])

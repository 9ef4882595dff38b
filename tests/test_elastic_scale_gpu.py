"""FP32 elastic plans: the traces of the one-thread-per-cell kernels and of the interior
strips are as near to the FP64 plan's as those of the row kernels, whose arithmetic has
the same storage and one rounding a field and step.  What can set them apart is a factor
of all differences (1/(24h) rounded to FP32 by itself: 5e-8 at h = 10), an error of the
wave speed, 1.2 to 1.4 times the row kernels' error over these records.  The bound, 1.2,
leaves room for another order of the same roundings."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# (NX, NY): cells alone, interior strips beside them
@pytest.mark.parametrize("NX,NY", [(331, 201), (620, 411)])
def test_fp32_plan_error_as_the_row_kernels(ads, cuda, NX, NY):
    T, n = 500, 20
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=T, DELTAX=10.0, DELTAY=10.0,
                                    DELTAT=0.7e-3, NPOINTS_PML=n, vp_ref=3000.0, f0=10.0)
    z = np.linspace(0, 1, NY + 2)[None, :] + np.zeros((NX + 2, 1))
    vp = 2500 + 2000 / (1 + np.exp(-30 * (z - 0.4)))
    model = [torch.as_tensor(a, dtype=torch.float64, device=cuda)
             for a in ads.compute_properties(vp, vp / 1.75, 310 * vp ** 0.25)]
    f = 10.0
    a = (np.pi * f * (np.arange(T) * p.DELTAT - 1.2 / f)) ** 2
    wav = (1e6 * (1 - 2 * a) * np.exp(-a))[:, None]
    xr = np.arange(n + 3, NX - n, 2)
    shots = [dict(srci=[s] * 2, srcj=[n + 9] * 2, srctype=[2, 3], srcv=np.repeat(wav, 2, 1),
                  rcvi=np.concatenate([xr, xr]), rcvj=np.full(2 * len(xr), n + 6),
                  rcvtype=np.repeat([0, 1], len(xr))) for s in (NX // 3, 2 * NX // 3)]
    if NX * NY < 200000:
        shots = shots[:1]

    def traces(precision, **kw):
        plan = ads.ElasticPlan(p, shots, precision=precision, **kw)
        out = plan.forward(*model).double().clone()
        plan.close()
        return out

    true = traces("f64")
    err = lambda t: float((t - true).norm() / true.norm())
    rows = traces("f32", rows_per_warp=8)
    assert err(traces("f32")) <= 1.2 * err(rows)

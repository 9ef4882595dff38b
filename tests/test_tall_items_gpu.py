"""Items of more rows than sixteen bits hold: a model of 40,000 rows with a row height
configured that gives an item 32,768 of them, against the oracle (1e-12, as the other
FP64 plans; FP32 1e-5 and 1e-4)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,variant", [("f64", 0), ("f64", 1), ("f32", 0), ("f32", 1)])
def test_tall_items(ads, orc, cuda, precision, variant):
    nx, ny, T, h, dt, npml, vref = 40000, 8, 5, 10.0, 1e-3, 2, 1500.0
    rng = np.random.default_rng(3)
    vp = 1800 + 900 * rng.random((nx + 2, ny + 2))
    sx, ty = orc.acoustic_pml(nx, ny, h, h, npml, vref)
    si = rng.integers(2, nx + 2, 60)
    si[:4] = 2, 32768, 32769, nx + 1
    sj = rng.integers(2, ny + 2, 60)
    srcv = rng.standard_normal((T, 60)) * 1e3
    ri, rj = si.copy(), np.full(60, 5)
    a = (nx, ny, T, dt, h, h, sx, ty, vp.reshape(-1), si, sj, srcv, ri, rj)
    tr = np.asarray(orc.acoustic_forward(*a, variant=variant)).reshape(T + 1, -1)
    loss, grad = orc.acoustic_gradient(*a, 0.9 * tr, variant=variant)
    shot = dict(x0=0, nx=nx, nstep=T, srci=si, srcj=sj, srcv=srcv, rcvi=ri, rcvj=rj)
    plan = ads.AcousticPlan(nx, ny, h, h, dt, [shot], npml=npml, vp_ref=vref, precision=precision,
                            variant=variant, rows_per_thread=8192, ckpt_every=3)
    rel = lambda x, y: np.linalg.norm(x - y) / np.linalg.norm(y)
    tol_tr, tol = (1e-12, 1e-12) if precision == "f64" else (1e-5, 1e-4)
    vt = torch.as_tensor(vp, dtype=torch.float64, device=cuda)
    assert rel(plan.forward(vt).double().cpu().numpy().reshape(T + 1, -1), tr) <= tol_tr
    l, g = plan.gradient(vt, torch.as_tensor(0.9 * tr.reshape(-1), device=cuda).to(plan.dtype))
    assert abs(float(l) - loss) <= tol * loss
    assert rel(g.cpu().numpy().reshape(-1), np.asarray(grad).reshape(-1)) <= tol
    plan.close()

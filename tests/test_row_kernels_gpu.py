"""The row-walking acoustic kernels where a plan's defaults no longer reach them on small
grids: configured row heights in FP64 variant U, FP32 variant U at the size where they
are the default, and the autotuner over them, against the oracle.

Tolerances as the other plan tests: FP64 1e-12, FP32 1e-5 traces and 1e-4 the rest."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

H, DT, VREF = 10.0, 1e-3, 1500.0


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64).reshape(-1), np.asarray(b, dtype=np.float64).reshape(-1)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def survey(orc, MX, MY, npml, windows, variant, seed, nsrc=3):
    """Shots of the windows (x0, nx, nstep), the model, and the oracle's answers."""
    rng = np.random.default_rng(seed)
    vp = 1800 + 900 * rng.random((MX + 2, MY + 2))
    shots, trs, obs, loss, grad = [], [], [], 0.0, np.zeros_like(vp)
    for x0, nx, t in windows:
        sx, ty = orc.acoustic_pml(nx, MY, H, H, npml, VREF)
        si, sj = rng.integers(2, nx + 2, nsrc), rng.integers(2, MY + 2, nsrc)
        si[0], sj[0] = nx // 2, npml + 9  # (one whose waves reach the receivers)
        srcv = rng.standard_normal((t, nsrc)) * 1e3
        ri = np.arange(2, nx + 2, 3)
        rj = np.full(len(ri), npml + 4)
        a = (nx, MY, t, DT, H, H, sx, ty, vp[x0:x0 + nx + 2].reshape(-1), si, sj, srcv, ri, rj)
        trs.append(np.asarray(orc.acoustic_forward(*a, variant=variant)).reshape(t + 1, -1))
        obs.append(0.9 * trs[-1] + 1e-3 * rng.standard_normal(trs[-1].shape))
        l, g = orc.acoustic_gradient(*a, obs[-1], variant=variant)
        loss += l
        grad[x0:x0 + nx + 2] += np.asarray(g).reshape(nx + 2, MY + 2)
        shots.append(dict(x0=x0, nx=nx, nstep=t, srci=si, srcj=sj, srcv=srcv, rcvi=ri, rcvj=rj))
    return shots, vp, trs, obs, loss, grad


def check(plan, cuda, vp, trs, obs, loss, grad, tol_tr, tol):
    vt = torch.as_tensor(vp, dtype=torch.float64, device=cuda)
    for a, b in zip(plan.split_traces(plan.forward(vt)), trs):
        assert rel(a.double().cpu().numpy(), b) <= tol_tr
    l, g = plan.gradient(vt, plan.pack([torch.as_tensor(o, device=cuda) for o in obs]))
    torch.cuda.synchronize()
    assert abs(float(l) - loss) <= tol * loss
    assert rel(g.cpu().numpy(), grad) <= tol


SMALL = ((0, 150, 60), (13, 101, 60), (40, 97, 47))


@pytest.fixture(scope="module")
def small(orc):
    return {v: survey(orc, 150, 190, 12, SMALL, v, 17 + v) for v in (0, 1)}


@pytest.mark.parametrize("rows,resident,graph", [(1, -1, True), (2, 1, False), (4, 0, True)])
def test_fp64_variant_u_rows(ads, cuda, small, rows, resident, graph):
    shots, vp, trs, obs, loss, grad = small[1]
    plan = ads.AcousticPlan(150, 190, H, H, DT, shots, npml=12, vp_ref=VREF, precision="f64",
                            variant=1, ckpt_every=13, rows_per_thread=rows,
                            resident_segments=resident, use_graph=graph)
    assert plan.rows == (rows,) * 4
    check(plan, cuda, vp, trs, obs, loss, grad, 1e-12, 1e-12)
    plan.close()


@pytest.mark.parametrize("precision,variant,kw", [("f64", 0, dict(rows_per_thread=2)),
                                                  ("f64", 1, dict(rows_per_thread=2)),
                                                  ("f32", 0, dict(rows_per_thread=2)),
                                                  ("f32", 1, dict(rows_per_thread=2)),
                                                  ("f32", 0, dict(steps_per_block=2)),
                                                  ("f32", 0, dict(tma=1))])
def test_autotuned_rows(ads, cuda, small, precision, variant, kw):
    """(a plan with configured rows, tensor maps or blocked steps keeps the row kernels,
    and its autotuner runs)"""
    shots, vp, trs, obs, loss, grad = small[variant]
    plan = ads.AcousticPlan(150, 190, H, H, DT, shots, npml=12, vp_ref=VREF, precision=precision,
                            variant=variant, ckpt_every=13, autotune=True, **kw)
    check(plan, cuda, vp, trs, obs, loss, grad, *((1e-12, 1e-12) if precision == "f64" else
                                                  (1e-5, 1e-4)))
    plan.close()


@pytest.mark.parametrize("autotune", [False, True])
def test_fp32_variant_u_of_a_million_cells(ads, orc, cuda, autotune):
    MX, MY = 700, 540
    shots, vp, trs, obs, loss, grad = survey(orc, MX, MY, 14, ((0, 700, 22), (0, 700, 22), (9, 680, 17)),
                                             1, 5)
    plan = ads.AcousticPlan(MX, MY, H, H, DT, shots, npml=14, vp_ref=VREF, precision="f32",
                            variant=1, ckpt_every=6, resident_segments=1, autotune=autotune)
    assert max(plan.rows) > 1  # (the cell kernels have 1 throughout)
    check(plan, cuda, vp, trs, obs, loss, grad, 1e-5, 1e-4)
    plan.close()

"""The acoustic one-thread-per-cell step kernels (FP64 plans, small FP32 plans) at
the grid sizes where their tiles (4 rows, strips of up to 32 columns with one narrow
strip) can go wrong: sources beside tile edges, more than a warp's width of
receivers in a tile, receivers that share a cell, two shots of unequal windows and
record lengths, recomputed and resident segments, both variants, against the
oracle.

Tolerances as the other plan tests take for loops of this length: FP64 1e-12,
FP32 1e-5 for traces and 1e-4 for loss and gradients."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2), (4, 31), (5, 33), (8, 32), (9, 66), (16, 97), (33, 40), (24, 130)]


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_cells_over_tile_edges(ads, orc, cuda, shape, precision, variant):
    NX, NY = shape
    hx, hy, dt, vref = 10.0, 8.0, 1e-3, 1500.0
    npml = max(1, min(NX, NY) // 4)
    rng = np.random.default_rng(NX * 1000 + NY + variant)
    vp = 1800 + 900 * rng.random((NX + 2, NY + 2))
    shots, ref_l, ref_g, obs, trs, gsrc = [], 0.0, np.zeros_like(vp), [], [], []
    for x0, nx, T in ((0, NX, 37), (NX // 3, NX - NX // 3, 29)):
        sx, ty = orc.acoustic_pml(nx, NY, hx, hy, npml, vref)
        si = np.unique(np.clip([2, 5, 9, 10, nx // 2 + 1, nx + 1], 2, nx + 1))
        sj = np.clip(rng.choice([2, 32, 33, 34, NY // 2 + 1, NY + 1], len(si)), 2, NY + 1)
        srcv = rng.standard_normal((T, len(si))) * 1e3
        # a block of receivers on every cell, and some cells again
        ri, rj = (a.reshape(-1) for a in np.meshgrid(np.arange(2, min(nx, 12) + 2),
                                                     np.arange(2, min(NY, 20) + 2)))
        ri, rj = np.concatenate([ri, ri[:5]]), np.concatenate([rj, rj[:5]])
        v = vp[x0:x0 + nx + 2]
        a = (nx, NY, T, dt, hx, hy, sx, ty, v.reshape(-1), si, sj, srcv, ri, rj)
        tr = np.asarray(orc.acoustic_forward(*a, variant=variant)).reshape(T + 1, -1)
        o = 0.9 * tr + 1e-3 * rng.standard_normal(tr.shape)
        l, g, gs = orc.acoustic_gradient(*a, o, variant=variant, want_src=True)
        ref_l += l
        ref_g[x0:x0 + nx + 2] += np.asarray(g).reshape(nx + 2, NY + 2)
        gsrc.append(np.asarray(gs).reshape(T, -1))
        trs.append(tr)
        obs.append(o)
        shots.append(dict(x0=x0, nx=nx, nstep=T, srci=si, srcj=sj, srcv=srcv, rcvi=ri, rcvj=rj))
    plan = ads.AcousticPlan(NX, NY, hx, hy, dt, shots, npml=npml, vp_ref=vref,
                            precision=precision, variant=variant, ckpt_every=9,
                            resident_segments=2)
    assert plan.rows == (1, 1, 1, 1)
    vt = torch.as_tensor(vp, dtype=torch.float64, device=cuda)
    tol, tol_tr = (1e-12, 1e-12) if precision == "f64" else (1e-4, 1e-5)
    for a, b in zip(plan.split_traces(plan.forward(vt)), trs):
        assert rel(a.double().cpu().numpy(), b) <= tol_tr
    loss, grad, gs = plan.gradient(vt, plan.pack([torch.as_tensor(o, device=cuda) for o in obs]),
                                   want_source_grad=True)
    torch.cuda.synchronize()
    assert abs(float(loss) - ref_l) <= tol * ref_l
    assert rel(grad.cpu().numpy(), ref_g) <= tol
    for a, b in zip(gs, gsrc):
        assert rel(a.cpu().numpy(), b) <= tol
    plan.close()

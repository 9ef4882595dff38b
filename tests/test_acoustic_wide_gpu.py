"""The larger FP32 acoustic plans (more cells than the one-thread-per-cell kernels
take): the four-column interior kernels beside the general ones, shots in groups,
against the oracle.  The grids cut the interior rectangle every way: damped on all
sides, on none, on one side of an axis; a last strip of four columns; a rectangle
that sources and receivers fall into; windows that are all damped; shots of one window
(whose tables are shared) and of several.

Tolerances as the other FP32 plan tests take: 1e-5 traces, 1e-4 loss and gradients
(rel-L2 against FP64)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# NY, npml, use_pml, variant: interior columns between the 64-column strips are
# 388 - 128 = 260 = 2 x 128 + 4, a leftover column past the rectangle, one-sided, ...
CASES = [(388, 12, 15, 0), (401, 30, 15, 0), (399, 12, 0, 0), (402, 12, 5, 0), (403, 12, 10, 0),
         (397, 70, 15, 0), (411, 12, 15, 1), (403, 12, 6, 1), (404, 12, 15, 2)]


@pytest.mark.parametrize("NY,npml,use_pml,variant", CASES)
def test_wide_plan_vs_oracle(ads, orc, cuda, NY, npml, use_pml, variant):
    # (variant U's plans reach these kernels at more cells and split into groups from
    # eight shots on; the last case, variant W, makes four groups, two a stream)
    MX, T, rep = {0: (330, 26, 1), 1: (600, 26, 3), 2: (560, 14, 8)}[variant]
    variant %= 2
    h, dt, vref = 10.0, 1e-3, 1500.0
    rng = np.random.default_rng(NY + use_pml)
    vp = 1800 + 900 * rng.random((MX + 2, NY + 2))
    nx2 = MX - 40
    shots, loss, grad, obs, trs, gsrc = [], 0.0, np.zeros_like(vp), [], [], []
    for x0, nx, t in rep * ((0, MX, T), (17, nx2, T), (23, nx2 - 3, T - 7)):
        sx, ty = orc.acoustic_pml(nx, NY, h, h, npml, vref, use_pml=use_pml)
        # sources in the rectangle, beside its edges, in the damped bands
        si = np.array([nx // 2, 2, nx + 1, nx // 3, npml + 2])
        sj = np.array([NY // 2, NY // 3, 70, 65, 2])
        srcv = rng.standard_normal((t, 5)) * 1e3
        ri = np.concatenate([np.arange(2, nx + 2, 7), np.full(40, nx // 2)])
        rj = np.concatenate([np.full(len(ri) - 40, npml + 4), np.linspace(2, NY + 1, 40).astype(int)])
        a = (nx, NY, t, dt, h, h, sx, ty, vp[x0:x0 + nx + 2].reshape(-1), si, sj, srcv, ri, rj)
        tr = np.asarray(orc.acoustic_forward(*a, variant=variant)).reshape(t + 1, -1)
        o = 0.9 * tr + 1e-3 * rng.standard_normal(tr.shape)
        l, g, gs = orc.acoustic_gradient(*a, o, variant=variant, want_src=True)
        loss += l
        grad[x0:x0 + nx + 2] += np.asarray(g).reshape(nx + 2, NY + 2)
        gsrc.append(np.asarray(gs).reshape(t, -1))
        trs.append(tr)
        obs.append(o)
        shots.append(dict(x0=x0, nx=nx, nstep=t, srci=si, srcj=sj, srcv=srcv, rcvi=ri, rcvj=rj))
    vt = torch.as_tensor(vp, dtype=torch.float64, device=cuda)
    for graph, resident, tune in ((True, 1, False), (False, -1, True)):
        plan = ads.AcousticPlan(MX, NY, h, h, dt, shots, npml=npml, vp_ref=vref, use_pml=use_pml,
                                precision="f32", variant=variant, ckpt_every=11,
                                resident_segments=resident, use_graph=graph, autotune=tune)
        assert min(plan.rows) > 1  # (not the one-thread-per-cell kernels)
        for a, b in zip(plan.split_traces(plan.forward(vt)), trs):
            assert rel(a.double().cpu().numpy(), b) <= 1e-5
        got, g, gs = plan.gradient(vt, plan.pack([torch.as_tensor(o, device=cuda) for o in obs]),
                                   want_source_grad=True)
        torch.cuda.synchronize()
        assert abs(float(got) - loss) <= 1e-4 * loss
        assert rel(g.cpu().numpy(), grad) <= 1e-4
        for a, b in zip(gs, gsrc):
            assert rel(a.cpu().numpy(), b) <= 1e-4
        plan.close()

"""FP64 plans of about half to all of the blocks that fit the chip at once, whose chained
launches let the next one start at their end, against the oracle.

Tolerances as the other FP64 plan tests: 1e-12 (rel-L2)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64).reshape(-1), np.asarray(b, dtype=np.float64).reshape(-1)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# one shot: 675 to 1125 blocks of 4 x 32 cells; the last pair's shorter record leaves one
# shot's blocks for its last steps
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("nx,ny,nshots", [(297, 260, 1), (500, 280, 1), (240, 200, 2)])
def test_acoustic(ads, orc, cuda, nx, ny, nshots, variant):
    T, h, dt, npml, vref = 40, 10.0, 1e-3, 14, 1500.0
    rng = np.random.default_rng(nx + variant)
    vp = 1800 + 900 * rng.random((nx + 2, ny + 2))
    sx, ty = orc.acoustic_pml(nx, ny, h, h, npml, vref)
    si, sj = np.array([nx // 2, 5, nx - 3]), np.array([ny // 2, 20, 9])
    ri = np.arange(2, nx + 2, 3)
    rj = np.full(len(ri), npml + 4)
    shots, obs, loss, grad, trs = [], [], 0.0, 0.0, []
    for k in range(nshots):
        t = T - 9 * k
        srcv = rng.standard_normal((t, 3)) * 1e3
        a = (nx, ny, t, dt, h, h, sx, ty, vp.reshape(-1), si, sj, srcv, ri, rj)
        trs.append(np.asarray(orc.acoustic_forward(*a, variant=variant)))
        obs.append((0.9 * trs[-1]).reshape(t + 1, -1))
        l, g = orc.acoustic_gradient(*a, obs[-1], variant=variant)
        loss, grad = loss + l, grad + np.asarray(g)
        shots.append(dict(x0=0, nx=nx, nstep=t, srci=si, srcj=sj, srcv=srcv, rcvi=ri, rcvj=rj))
    plan = ads.AcousticPlan(nx, ny, h, h, dt, shots, npml=npml, vp_ref=vref, precision="f64",
                            variant=variant, ckpt_every=11, resident_segments=1)
    vt = torch.as_tensor(vp, dtype=torch.float64, device=cuda)
    for a, b in zip(plan.split_traces(plan.forward(vt)), trs):
        assert rel(a.cpu().numpy(), b) <= 1e-12
    l, g = plan.gradient(vt, plan.pack([torch.as_tensor(o, device=cuda) for o in obs]))
    assert abs(float(l) - loss) <= 1e-12 * loss
    assert rel(g.cpu().numpy(), grad) <= 1e-12
    plan.close()


# 192 and 1100 blocks of 8 x 32 cells
@pytest.mark.parametrize("NX,NY,nshots", [(253, 187, 1), (397, 350, 2)])
def test_elastic(ads, orc, cuda, NX, NY, nshots):
    T = 12
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=T, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=0.7e-3, NPOINTS_PML=11, vp_ref=3000.0, f0=15.0)
    ax, bx, kx, ay, by, ky = [a.reshape(-1) for a in ads.compute_elastic_PML_Params(p)]
    rng = np.random.default_rng(NX)
    vp = 3000 + 300 * rng.random((NX + 2, NY + 2))
    lam, mu, rho = [a.reshape(-1) for a in ads.compute_properties(
        vp, vp / 1.8, 2000 + 200 * rng.random((NX + 2, NY + 2)))]
    shots, obs, trs, ref = [], [], [], None
    for _ in range(nshots):
        src = (rng.integers(3, NX + 1, 200), rng.integers(3, NY + 1, 200), rng.integers(0, 5, 200),
               rng.standard_normal((T, 200)) * 1e3)
        rcv = (rng.integers(2, NX + 1, 300), rng.integers(2, NY + 1, 300), rng.integers(0, 5, 300))
        a = (NX, NY, T, p.DELTAT, p.DELTAX, p.DELTAY, ax, bx, ay, by, lam, mu, rho, *src, *rcv)
        trs.append(np.asarray(orc.elastic_forward(*a)).reshape(-1))
        obs.append(0.9 * trs[-1])
        g = orc.elastic_gradient(*a, obs[-1].reshape(300, T + 1))
        ref = g if ref is None else [x + y for x, y in zip(ref, g)]
        shots.append(dict(srci=src[0], srcj=src[1], srctype=src[2], srcv=src[3], rcvi=rcv[0],
                          rcvj=rcv[1], rcvtype=rcv[2]))
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=cuda)
    plan = ads.ElasticPlan(p, shots, precision="f64", ckpt_every=5)
    model = [t(lam), t(mu), t(rho)]
    assert rel(plan.forward(*model).cpu().numpy(), np.concatenate(trs)) <= 1e-12
    got = plan.gradient(*model, t(np.concatenate(obs)))
    for a, b in zip(got, ref):
        assert rel(a.cpu().numpy(), b) <= 1e-12
    plan.close()

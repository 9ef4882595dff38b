"""The FP32 elastic plans of middle size (interior strips beside one-thread-per-cell
tiles) and of several larger shots (row kernels, the shots in two halves), against the
oracle.  The grids cut the interior every way: strips of full and of odd width, a row
count that is no multiple of a block's, hardly any interior, none.

Tolerance 1e-4 (rel-L2 against FP64) as the other FP32 loops of this length."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# NX, NY, npml, shots (more than 200 000 cells in all; the last two more than 1.1 and 1.5 million)
CASES = [(330, 331, 10, 2), (353, 300, 30, 2), (1701, 61, 5, 2), (2700, 40, 4, 2),
         (101, 1033, 9, 2), (457, 161, 12, 3), (1190, 310, 5, 3), (1101, 700, 8, 2)]


@pytest.mark.parametrize("NX,NY,npml,nshots", CASES)
def test_plans_against_the_oracle(ads, orc, cuda, NX, NY, npml, nshots):
    T, tol = 11, 1e-4
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=T, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=0.7e-3, NPOINTS_PML=npml, vp_ref=3000.0, f0=15.0)
    ax, bx, kx, ay, by, ky = [a.reshape(-1) for a in ads.compute_elastic_PML_Params(p)]
    rng = np.random.default_rng(NX * 100 + NY)
    vp = 3000 + 300 * rng.random((NX + 2, NY + 2))
    lam, mu, rho = [a.reshape(-1) for a in ads.compute_properties(
        vp, vp / 1.8, 2000 + 200 * rng.random((NX + 2, NY + 2)))]
    shots, ref, obs_all, tr_all = [], None, [], []
    for _ in range(nshots):
        srci, srcj = rng.integers(3, NX + 1, 400), rng.integers(3, NY + 1, 400)
        srct, srcv = rng.integers(0, 5, 400), rng.standard_normal((T, 400)) * 1e3
        rcvi, rcvj = rng.integers(2, NX + 1, 700), rng.integers(2, NY + 1, 700)
        rcvt = rng.integers(0, 5, 700)
        a = (NX, NY, T, p.DELTAT, p.DELTAX, p.DELTAY, ax, bx, ay, by, lam, mu, rho, srci, srcj,
             srct, srcv, rcvi, rcvj, rcvt)
        tr = np.asarray(orc.elastic_forward(*a))
        obs = (tr + rng.standard_normal(tr.shape) * np.abs(tr).max()).reshape(700, T + 1)
        tr_all.append(tr.reshape(-1))
        g = orc.elastic_gradient(*a, obs)
        ref = g if ref is None else [x + y for x, y in zip(ref, g)]
        obs_all.append(obs.reshape(-1))
        shots.append(dict(srci=srci, srcj=srcj, srctype=srct, srcv=srcv, rcvi=rcvi, rcvj=rcvj,
                          rcvtype=rcvt))
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=cuda)
    for graph in (True, False):
        plan = ads.ElasticPlan(p, shots, precision="f32", ckpt_every=4, resident_segments=1,
                               use_graph=graph)
        tr = plan.forward(t(lam), t(mu), t(rho))
        assert rel(tr.cpu().numpy(), np.concatenate(tr_all)) <= tol
        loss, *grads = plan.gradient(t(lam), t(mu), t(rho), t(np.concatenate(obs_all)))
        torch.cuda.synchronize()
        assert abs(float(loss) - ref[0]) <= tol * ref[0]
        for a, b in zip(grads, ref[1:]):
            assert rel(a.cpu().numpy(), b) <= tol
        plan.close()

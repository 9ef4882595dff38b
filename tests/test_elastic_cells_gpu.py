"""The elastic one-thread-per-cell kernels at the sizes where their tiles (8 rows
x 32 columns) can go wrong, against the oracle: the single-step operators and the
plans that step with them (FP64, and FP32 below the row kernels' sizes).

Tolerances: one step and its transpose, 1e-13 (FP64 rounding of sums of some
twenty products, 2^-53 each; FP32 the same with 2^-24: 1e-5).  A plan's loop of T
steps carries a rounding of each step on: 1e-12 as the other FP64 plan tests
take for loops of this length, 1e-4 for FP32."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# below, on and beyond the tiles' edges (cells 1..N in plans, 0..N+1 in operators)
SIZES = [(4, 4), (6, 30), (7, 31), (8, 32), (9, 33), (33, 65)]
PLAN_SIZES = [(8, 4), (8, 32), (9, 33), (15, 31), (16, 63), (33, 65)]  # (plans take NX >= 8)


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def problem(ads, NX, NY, T=1):
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=T, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=0.7e-3, NPOINTS_PML=max(1, min(NX, NY) // 4),
                                    vp_ref=3000.0, f0=15.0)
    prof = ads.compute_elastic_PML_Params(p)
    rng = np.random.default_rng(NX * 100 + NY)
    vp = 3000 + 300 * rng.random((NX + 2, NY + 2))
    lam, mu, rho = ads.compute_properties(vp, vp / 1.8, 2000 + 200 * rng.random((NX + 2, NY + 2)))
    return p, prof, [a.reshape(-1) for a in (lam, mu, rho)], rng


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 1e-5)])
@pytest.mark.parametrize("shape", SIZES)
def test_operators_over_tile_edges(ads, orc, cuda, shape, dtype, tol):
    NX, NY = shape
    N = (NX + 2) * (NY + 2)
    p, prof, model, rng = problem(ads, NX, NY)
    rd = lambda a: torch.as_tensor(np.asarray(a), dtype=dtype).double().numpy()
    ax, bx, kx, ay, by, ky = [rd(a).reshape(-1) for a in prof]
    lam, mu, rho = (rd(a) for a in model)
    st, w = rd(rng.standard_normal(13 * N)), rd(rng.standard_normal(13 * N))
    src = ([NX // 2 + 1, 2], [NY // 2 + 1, 3], [2, 0], rd([1.5, -2.0]))
    k = (p.DELTAT, p.DELTAX, p.DELTAY, NX, NY)
    ref = orc.elastic_step_fwd(st, lam, mu, rho, ax, bx, ay, by, *k, *src)
    refg = orc.elastic_step_bwd(st, w, lam, mu, rho, ax, bx, ay, by, *k)
    t = lambda a: torch.as_tensor(np.asarray(a), dtype=dtype, device=cuda)
    args = (p, t(rho), t(lam), t(mu), t(st).view(13, N))
    tp = [t(a) for a in prof]
    got = ads.elastic_one_step(*args, tp, src[0], src[1], src[3], src[2])
    assert rel(got.double().cpu().numpy().reshape(-1), ref) <= tol
    gotg = ads.elastic_one_step_grad(*args, t(w).view(13, N), tp)
    for a, b in zip(gotg, refg):
        assert rel(a.double().cpu().numpy().reshape(-1), b) <= tol


@pytest.mark.parametrize("name", ["ads_elastic_step_bwd_f64", "ads_elastic_step_bwd_f64_noalloc"])
def test_transpose_into_the_state_array(ads, orc, cuda, name):
    """grad_in may be state_in itself: the step is taken about the old values."""
    from adseismic_gb300._lib import call

    NX, NY = 19, 37
    N = (NX + 2) * (NY + 2)
    p, prof, (lam, mu, rho), rng = problem(ads, NX, NY)
    ax, bx, kx, ay, by, ky = [a.reshape(-1) for a in prof]
    st, w = rng.standard_normal(13 * N), rng.standard_normal(13 * N)
    k = (p.DELTAT, p.DELTAX, p.DELTAY, NX, NY)
    ref = orc.elastic_step_bwd(st, w, lam, mu, rho, ax, bx, ay, by, *k)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=cuda)
    s = t(st)
    g = [torch.zeros(N, dtype=torch.float64, device=cuda) for _ in range(3)]
    ins = [s, t(w), s, *g] + [t(a) for a in (lam, mu, rho, ax, bx, ay, by)]
    call(name, *[C.c_void_p(v.data_ptr()) for v in ins], *k,
         C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    for a, b in zip([s] + g, ref):
        assert rel(a.cpu().numpy(), b) <= 1e-13


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_operators_pass_on_values_that_are_not_finite(ads, orc, cuda, bad):
    """One such value in the state or in the output's gradient, where the CPML is
    idle: the same cells of every output are not finite."""
    NX, NY = 40, 70
    N = (NX + 2) * (NY + 2)
    p, prof, (lam, mu, rho), rng = problem(ads, NX, NY)
    p.NPOINTS_PML = 5
    prof = ads.compute_elastic_PML_Params(p)
    ax, bx, kx, ay, by, ky = [a.reshape(-1) for a in prof]
    k = (p.DELTAT, p.DELTAX, p.DELTAY, NX, NY)
    t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=cuda)
    for f in range(13):
        st, w = rng.standard_normal(13 * N), rng.standard_normal(13 * N)
        at = f * N + 16 * (NY + 2) + 33
        with np.errstate(all="ignore"):
            a = st.copy()
            a[at] = bad
            ref = orc.elastic_step_fwd(a, lam, mu, rho, ax, bx, ay, by, *k)
            got = ads.elastic_one_step(p, t(rho), t(lam), t(mu), t(a).view(13, N), prof)
            assert np.array_equal(np.isfinite(got.cpu().numpy().reshape(-1)), np.isfinite(ref)), f
            b = w.copy()
            b[at] = bad
            refg = orc.elastic_step_bwd(st, b, lam, mu, rho, ax, bx, ay, by, *k)
            gotg = ads.elastic_one_step_grad(p, t(rho), t(lam), t(mu), t(st).view(13, N),
                                             t(b).view(13, N), prof)
        for x, y in zip(gotg, refg):
            assert np.array_equal(np.isfinite(x.cpu().numpy().reshape(-1)), np.isfinite(y)), f


@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-4)])
@pytest.mark.parametrize("shape", PLAN_SIZES)
def test_plans_over_tile_edges(ads, orc, cuda, shape, precision, tol):
    """Two shots, an odd checkpoint spacing with recomputed and resident segments."""
    NX, NY = shape
    T = 23
    p, prof, (lam, mu, rho), rng = problem(ads, NX, NY, T)
    ax, bx, kx, ay, by, ky = [a.reshape(-1) for a in prof]
    shots, ref, obs_all, tr_all = [], None, [], []
    for _ in range(2):
        srci, srcj = rng.integers(3, NX + 1, 4), rng.integers(3, NY + 1, 4)
        srct, srcv = np.array([0, 1, 2, 4]), rng.standard_normal((T, 4)) * 1e3
        rcvi, rcvj = rng.integers(2, NX + 1, 9), rng.integers(2, NY + 1, 9)
        rcvt = rng.integers(0, 5, 9)
        obs = rng.standard_normal((9, T + 1)) * 1e-3
        a = (NX, NY, T, p.DELTAT, p.DELTAX, p.DELTAY, ax, bx, ay, by, lam, mu, rho, srci, srcj,
             srct, srcv, rcvi, rcvj, rcvt)
        tr_all.append(np.asarray(orc.elastic_forward(*a)).reshape(-1))
        g = orc.elastic_gradient(*a, obs)
        ref = g if ref is None else [x + y for x, y in zip(ref, g)]
        obs_all.append(obs.reshape(-1))
        shots.append(dict(srci=srci, srcj=srcj, srctype=srct, srcv=srcv, rcvi=rcvi, rcvj=rcvj,
                          rcvtype=rcvt))
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=cuda)
    plan = ads.ElasticPlan(p, shots, precision=precision, ckpt_every=7, resident_segments=1)
    tr = plan.forward(t(lam), t(mu), t(rho))
    assert rel(tr.cpu().numpy(), np.concatenate(tr_all)) <= tol
    loss, *grads = plan.gradient(t(lam), t(mu), t(rho), t(np.concatenate(obs_all)))
    torch.cuda.synchronize()
    assert abs(float(loss) - ref[0]) <= tol * ref[0]
    for a, b in zip(grads, ref[1:]):
        assert rel(a.cpu().numpy(), b) <= tol
    plan.close()

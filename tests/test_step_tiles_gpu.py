"""The acoustic single-step kernels at the sizes where their tiles can go wrong
(one cell, tile edges and remainders) with the PML's mix of damped and undamped
cells, and their treatment of values that are not finite, against the oracle.

Tolerances: the forward performs the oracle's own operations in its order
(variant W bit for bit); the transpose sums at most 12 products per cell in
another order and with fused multiply-adds, so it differs by a few units in
the last place (2^-53) of its largest terms: 1e-14 in rel-L2."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def inputs(orc, NX, NY, seed):
    rng = np.random.default_rng(seed)
    N = (NX + 2) * (NY + 2)
    sx, ty = orc.acoustic_pml(NX, NY, 10.0, 8.0, 9, 1500.0)
    sig = np.repeat(sx[:, None], NY + 2, axis=1).reshape(-1)
    tau = np.repeat(ty[None, :], NX + 2, axis=0).reshape(-1)
    w, wo, p, q = (rng.standard_normal(N) for _ in range(4))
    c = (1500.0 + 2500.0 * rng.random(N)) ** 2
    return [w, wo, p, q, sig, tau, c], [rng.standard_normal(N) for _ in range(3)]


def both(ads, orc, cuda, ins, gs, NX, NY, variant):
    k = (1e-3, 10.0, 8.0, NX, NY)
    T = lambda x: torch.as_tensor(np.asarray(x), dtype=torch.float64, device=cuda)
    ref = orc.acoustic_step_fwd(*ins, *k, variant=variant)
    got = ads.acoustic_one_step(*[T(x) for x in ins], *k, variant)
    refg = orc.acoustic_step_bwd(*gs, *ins, *k, *ref, variant=variant)
    gotg = ads.acoustic_one_step_grad(*[T(x) for x in gs], *[T(x) for x in ins], *k,
                                      *[T(x) for x in ref], variant)
    n = lambda ts: [t.cpu().numpy() for t in ts]
    return n(got), [np.asarray(a) for a in ref], n(gotg), [np.asarray(a) for a in refg]


# (NX + 2, NY + 2) below, on and beyond tiles of 8 rows x 32 columns
SIZES = [(1, 1), (5, 29), (6, 30), (7, 31), (30, 62), (31, 63), (64, 33), (257, 301)]


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("shape", SIZES)
def test_step_and_transpose_over_tile_edges(ads, orc, cuda, shape, variant):
    NX, NY = shape
    ins, gs = inputs(orc, NX, NY, NX + NY + variant)
    got, ref, gotg, refg = both(ads, orc, cuda, ins, gs, NX, NY, variant)
    for a, b in zip(got, ref):
        if variant == 0:
            assert np.array_equal(a, b)
        else:
            assert rel(a, b) <= 1e-15
    for a, b in zip(gotg, refg):
        assert rel(a, b) <= 1e-14


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_not_finite_values_reach_the_same_cells(ads, orc, cuda, variant, bad):
    """One such value in each input (undamped cells, beside a tile's edge and
    on it): the same cells of every output are NaN, infinite or finite, and the
    forward's values agree to the bit, signed zeros included."""
    NX, NY = 62, 70
    for which in range(7):
        ins, gs = inputs(orc, NX, NY, 3)
        for a in ins[:4]:
            a[::3] = -0.0
        at = (31 if which % 2 else 32) * (NY + 2) + 32
        if which < 4:
            ins[which][at] = bad
        else:
            gs[which - 4][at] = bad
        with np.errstate(all="ignore"):
            got, ref, gotg, refg = both(ads, orc, cuda, ins, gs, NX, NY, variant)
        for a, b in zip(got, ref):
            assert np.array_equal(np.isnan(a), np.isnan(b)), which
            m = ~np.isnan(b)
            if variant == 0:
                assert np.array_equal(a[m].view(np.int64), b[m].view(np.int64)), which
        for a, b in zip(gotg, refg):
            assert np.array_equal(np.isnan(a), np.isnan(b)), which
            assert np.array_equal(np.isinf(a), np.isinf(b)), which

"""elastic_one_step's sources from host values (kernel arguments, 64 a launch) against the
same values on the device: the same additions in the same order, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nsrc", [1, 63, 64, 65, 130])
def test_host_and_device_values(ads, cuda, nsrc, dtype):
    NX, NY = 9, 14
    N = (NX + 2) * (NY + 2)
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=1, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=0.7e-3, NPOINTS_PML=2, vp_ref=3000.0, f0=15.0)
    prof = ads.compute_elastic_PML_Params(p)
    rng = np.random.default_rng(nsrc)
    t = lambda a: torch.as_tensor(a, dtype=dtype, device=cuda)
    lam, mu, rho = (t(1e9 + 1e8 * rng.random(N)) for _ in range(3))
    args = (p, rho, lam, mu, t(rng.standard_normal((13, N))), prof)
    # cells on the frame and outside the grid, types that do not exist, repeated cells
    si, sj = rng.integers(0, NX + 4, nsrc), rng.integers(0, NY + 4, nsrc)
    st, v = rng.integers(-1, 7, nsrc), rng.standard_normal(nsrc)
    a = ads.elastic_one_step(*args, si, sj, v, st)
    b = ads.elastic_one_step(*args, si, sj, torch.as_tensor(v, device=cuda), st)
    c = ads.elastic_one_step(*args, list(si), list(sj), torch.as_tensor(v), list(st))
    assert torch.equal(a, b) and torch.equal(a, c)
    with pytest.raises(ValueError):
        ads.elastic_one_step(*args, si, sj, v[:-1], st)

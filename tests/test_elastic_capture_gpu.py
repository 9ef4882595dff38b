"""elastic_one_step under stream capture refuses source values on the host: a graph would
add the values of the capture on each replay."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_sources_under_capture(ads, cuda):
    NX, NY = 40, 33
    N = (NX + 2) * (NY + 2)
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=1, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=1e-3, NPOINTS_PML=6, vp_ref=3000.0, f0=15.0)
    t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=cuda)
    prof = [t(a) for a in ads.compute_elastic_PML_Params(p)]
    rng = np.random.default_rng(4)
    st = t(rng.standard_normal((13, N)))
    rho, lam, mu = (t(1 + rng.random(N)) for _ in range(3))
    si, sj, sv, ty = [9, 12], [8, 8], t([1.5, -2.0]), [2, 3]
    step = lambda v: ads.elastic_one_step(p, rho, lam, mu, st, prof, si, sj, v, ty)
    want = step(sv)
    assert torch.equal(step(sv.cpu().numpy()), want)
    torch.cuda.synchronize()
    graph, host = torch.cuda.CUDAGraph(), sv.cpu().numpy()
    with pytest.raises(RuntimeError, match="cannot be captured"):
        with torch.cuda.graph(graph):
            step(host)
    torch.cuda.synchronize()
    assert torch.equal(step(sv), want)

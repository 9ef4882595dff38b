"""Source values of the single-step elastic operator in every form it takes them from the
host: arrays, lists, tensors of any floating type, tensors that require a gradient, and
lists of numbers that are tensors themselves."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_forms_of_source_values(ads, cuda, dtype):
    NX, NY = 30, 29
    N = (NX + 2) * (NY + 2)
    p = ads.ElasticPropagatorParams(NX=NX, NY=NY, NSTEP=1, DELTAX=10.0, DELTAY=8.0,
                                    DELTAT=1e-3, NPOINTS_PML=5, vp_ref=3000.0, f0=15.0)
    t = lambda a: torch.as_tensor(np.asarray(a), dtype=dtype, device=cuda)
    prof = [t(a) for a in ads.compute_elastic_PML_Params(p)]
    rng = np.random.default_rng(4)
    st = t(rng.standard_normal((13, N)))
    model = [t(1 + rng.random(N)) for _ in range(3)]
    vals = [1.5, -2.25]  # (exact in every type below)
    step = lambda v: ads.elastic_one_step(p, *model, st, prof, [9, 12], [8, 8], v, [2, 3])
    want = step(t(vals))
    forms = [vals, tuple(vals), np.array(vals), np.array(vals, np.float32), np.array([[1.5], [-2.25]]),
             torch.tensor(vals, dtype=torch.float64, requires_grad=True),
             [torch.tensor(v) for v in vals], [torch.tensor(v, device=cuda) for v in vals]]
    forms += [torch.tensor(vals, dtype=d) for d in (torch.float32, torch.float16, torch.bfloat16)]
    for v in forms:
        assert torch.equal(step(v), want)

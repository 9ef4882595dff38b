"""The FP64 acoustic forward operator performs the reference's own operations in its
order, so it agrees with the oracle bit for bit: in variant U too, whose coefficients the
reference forms in another order than variant W's, and for steps and spacings where the
two orders round apart."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("dt,hx,hy", [(1e-3, 10.0, 8.0), (0.7e-3, 12.5, 10.0), (0.9e-3, 7.0, 11.0),
                                      (1.1e-3, 20.0, 12.0), (0.8e-3, 13.0, 9.1)])
def test_forward_bits(ads, orc, cuda, dt, hx, hy, variant):
    NX, NY = 70, 61
    rng = np.random.default_rng(int(hx * 10))
    N = (NX + 2) * (NY + 2)
    sig, tau = (np.asarray(a) for a in orc.acoustic_pml(NX, NY, hx, hy, 9, 1500.0))
    ins = [rng.standard_normal(N) for _ in range(4)] + [sig, tau, (1500 + 2500 * rng.random(N)) ** 2]
    ref = orc.acoustic_step_fwd(*ins, dt, hx, hy, NX, NY, variant=variant)
    got = ads.acoustic_one_step(*[torch.as_tensor(a, device=cuda) for a in ins], dt, hx, hy, NX, NY,
                                variant)
    for a, b in zip(got, ref):
        assert np.array_equal(a.cpu().numpy(), np.asarray(b))

"""Plans bound the nodes of their graphs.

A plan of large shots and long records has as many groups of shots as keep its fields in
L2; each group's steps are nodes of their own.  Where that passes the limit, the plan has
fewer groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 400000


@pytest.mark.parametrize("variant", [0, 1])
def test_fewer_groups_beyond_the_limit(ads, cuda, variant):
    # eight groups' worth of live fields (variant U: six) over 12,000 steps: twice the limit
    nx, ny, T, n = 1000, 1990, 12000, 8
    shots = [dict(x0=0, nx=nx, nstep=T - 3 * k, srci=[nx // 2 + k], srcj=[40],
                  srcv=np.ones((T, 1)), rcvi=[100, 500], rcvj=[30, 30]) for k in range(n)]
    plan = ads.AcousticPlan(nx, ny, 10.0, 10.0, 1e-3, shots, npml=20, vp_ref=1500.0,
                            precision="f32", variant=variant, ckpt_every=250,
                            resident_segments=-1)
    # (a node a launch; what a segment adds to its steps' kernels is below 2%)
    assert plan.launches_gradient <= 1.02 * LIMIT
    plan.close()

"""Which kernels an FP32 acoustic plan in variant U takes below a million cells: the ones
that take less time a step, by the plan's damped and free rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# wide layers and many shots: the row kernels are ahead; one large shot, thin layers: not
@pytest.mark.parametrize("nx,ny,nshots,npml,cells", [(320, 300, 10, 40, False),
                                                     (425, 429, 4, 40, False),
                                                     (500, 400, 4, 12, True),
                                                     (1000, 700, 1, 40, True)])
def test_kernels_of_variant_u_fp32(ads, cuda, nx, ny, nshots, npml, cells):
    shot = dict(x0=0, nx=nx, nstep=6, srci=[nx // 2], srcj=[npml + 9], srcv=np.ones((6, 1)),
                rcvi=np.arange(npml, nx - npml), rcvj=np.full(nx - 2 * npml, npml + 5))
    plan = ads.AcousticPlan(nx, ny, 10.0, 10.0, 1e-3, [shot] * nshots, npml=npml, vp_ref=1500.0,
                            precision="f32", variant=1, resident_segments=-1)
    assert (max(plan.rows) == 1) == cells
    plan.close()

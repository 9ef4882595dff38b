"""autotune = 2 of FP32 acoustic plans: 2 and 4 forward steps a launch against the kernels
that the plan has by default, whatever its size, with answers held to the oracle (1e-5
traces, 1e-4 the rest)."""
import pytest

from test_row_kernels_gpu import DT, H, VREF, check, survey

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resident", [-1, 0])
def test_autotune_2_keeps_the_larger_plans_kernels(ads, orc, cuda, resident):
    """autotune = 2 times 2 and 4 steps a launch against the kernels the plan has, and does
    not give those up for the trial: on this size they win, so the plan is the one that
    autotune = 1 makes, groups of shots included (two: twice one group's launches)."""
    MX, MY = 1000, 320
    shots, vp, trs, obs, loss, grad = survey(orc, MX, MY, 14, 6 * ((0, 1000, 24),), 0, 3)
    launches = []
    for tune in (1, 2):
        plan = ads.AcousticPlan(MX, MY, H, H, DT, shots, npml=14, vp_ref=VREF, precision="f32",
                                ckpt_every=6, resident_segments=resident, autotune=tune)
        assert plan.steps_per_block == 1 and min(plan.rows) > 1
        launches.append(plan.launches_gradient)
        check(plan, cuda, vp, trs, obs, loss, grad, 1e-5, 1e-4)
        plan.close()
    assert launches[0] == launches[1]


@pytest.mark.parametrize("nx,ny", [(60, 50), (240, 200)])
def test_autotune_2_on_small_plans(ads, orc, cuda, nx, ny):
    """Small plans time blocked steps too; whichever wins, the answers hold."""
    shots, vp, trs, obs, loss, grad = survey(orc, nx, ny, 9, 2 * ((0, nx, 60),), 0, 8)
    plan = ads.AcousticPlan(nx, ny, H, H, DT, shots, npml=9, vp_ref=VREF, precision="f32",
                            ckpt_every=13, resident_segments=-1, autotune=2)
    assert plan.steps_per_block in (1, 2, 4)
    check(plan, cuda, vp, trs, obs, loss, grad, 1e-5, 1e-4)
    plan.close()

"""Single-step elastic operators on grids longer than a launch has blocks along its second
axis, in either direction: at both ends they give what a short grid of the same cells does,
to the bit (the same operations; the wave has not come in from the cut)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NX,NY", [(4, 65535 * 32 + 50), (65535 * 8 + 20, 4)])
def test_both_ends(ads, cuda, NX, NY):
    along = 0 if NX > NY else 1
    g = torch.Generator(device=cuda).manual_seed(5)
    shape = (NX + 2, NY + 2)
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float32, device=cuda)
    st, w = (rnd(13, *shape) - 0.5 for _ in range(2))
    model = [1 + rnd(*shape) for _ in range(3)]
    prof = []
    for n in (NX, NY):
        prof += [0.1 * rnd(2, n) - 0.1, 1 - 0.1 * rnd(2, n), torch.ones(2, n, device=cuda)]

    def run(nx, ny, st, w, model, prof):
        p = ads.ElasticPropagatorParams(NX=nx, NY=ny, NSTEP=1, DELTAX=10.0, DELTAY=8.0,
                                        DELTAT=1e-3, NPOINTS_PML=1, vp_ref=3000.0, f0=15.0)
        f = lambda a: a.reshape(13, -1).contiguous()
        m = [a.reshape(-1).contiguous() for a in model]
        out = ads.elastic_one_step(p, m[0], m[1], m[2], f(st), prof, [2], [2], [1.0], [2])
        gr = ads.elastic_one_step_grad(p, m[0], m[1], m[2], f(st), f(w), prof)
        return [a.reshape(-1, nx + 2, ny + 2) for a in (out, *gr)]

    full = run(NX, NY, st, w, model, prof)
    n, keep = 60, 40  # a short grid's length, and what of it is far from the cut
    for last in (False, True):
        cut = slice(-n - 2, None) if last else slice(0, n + 2)
        side = slice(-keep, None) if last else slice(0, keep)
        at = (lambda a, s: a[..., s, :]) if along == 0 else (lambda a, s: a[..., s])
        pr = [a[:, -n:].contiguous() if last else a[:, :n].contiguous() for a in prof]
        pr = pr[:3] + prof[3:] if along == 0 else prof[:3] + pr[3:]
        nx, ny = (n, NY) if along == 0 else (NX, n)
        part = run(nx, ny, at(st, cut), at(w, cut), [at(a, cut) for a in model], pr)
        for a, b in zip(full, part):  # (the source of the short grid lies far from its end)
            assert torch.equal(at(a, side), at(b, side))

"""Where the larger FP32 acoustic plans cut their undamped rectangle, and those plans
against the oracle where its right edge has no column to spare.

The rectangle's kernels know no damping, so no column of it may be damped or lie beside
a damped one; its first and last columns are multiples of four apart from column 1."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "wide_split.h"
extern "C" void split(int ny, const double* tau, int* out) {
  int nl, nr;
  ads::damped_runs(std::vector<double>(tau, tau + ny + 2), ny, nl, nr);
  ads::wide_columns(ny, nl, nr, out[0], out[1]);
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "split.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "adseismic.jl_gb300", "csrc"), str(d / "split.cpp"),
                    "-o", str(d / "split.so")], check=True)
    return ctypes.CDLL(str(d / "split.so")).split


@pytest.mark.parametrize("use_pml", [15, 0, 4, 8])
@pytest.mark.parametrize("npml", [1, 12, 30, 40, 61, 62, 63, 64, 65, 126, 127, 128, 129])
def test_no_damped_column_in_the_rectangle(split, orc, npml, use_pml):
    for ny in list(range(297, 305)) + [100, 131, 511, 512, 601, 602, 603]:
        tau = np.asarray(orc.acoustic_pml(40, ny, 10.0, 10.0, npml, 1500.0, use_pml=use_pml)[1])
        tau = np.ascontiguousarray(tau[:ny + 2], dtype=np.float64)
        out = (ctypes.c_int * 2)()
        split(ny, tau.ctypes.data_as(ctypes.c_void_p), out)
        jl, jr = out
        assert jl % 4 == 1 and jr % 4 == 1 and jl >= 1 and jr <= ny + 1
        for j in range(jl, jr):
            assert not tau[j - 1:j + 2].any(), (ny, j)
        # and it leaves at most one strip's width (and a rounding) of undamped columns out
        free = [j for j in range(1, ny + 1) if not tau[j - 1:j + 2].any()]
        if jr > jl:
            assert jl - free[0] < 64 and free[-1] - (jr - 1) < 64


# NY, npml, variant: right edges whose strips hold no, one or two undamped columns
EDGES = [(301, 64, 0), (302, 63, 0), (301, 62, 0), (305, 64, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("NY,npml,variant", EDGES)
def test_tight_right_edge_vs_oracle(ads, orc, cuda, NY, npml, variant):
    """A strong profile (vp_ref 1e5) damps even its first columns by parts in a
    thousand over the record; sources and receivers lie to the right of the rectangle.
    With one damped column taken for an undamped one the traces are 1e-4 off."""
    # enough cells that the plan takes the wide kernels (variant U from 1.6 M on)
    nx, T, rep = (400, 60, 3) if variant == 0 else (700, 60, 8)
    h, dt, vref = 10.0, 1e-3, 1e5
    rng = np.random.default_rng(NY + npml)
    vp = 2500 + 500 * rng.random((nx + 2, NY + 2))
    sx, ty = orc.acoustic_pml(nx, NY, h, h, npml, vref)
    edge = NY - npml  # (1-based padded index of the last undamped column)
    si = np.arange(100, nx - 80, 45)
    sj = np.full(len(si), edge + 8)
    srcv = rng.standard_normal((T, len(si))) * 1e3
    ri = np.arange(90, nx - 70, 3)
    rj = np.full(len(ri), edge + 6)
    a = (nx, NY, T, dt, h, h, sx, ty, vp.reshape(-1), si, sj, srcv, ri, rj)
    tr = np.asarray(orc.acoustic_forward(*a, variant=variant)).reshape(T + 1, -1)
    obs = 0.9 * tr
    loss, grad = orc.acoustic_gradient(*a, obs, variant=variant)
    shot = dict(x0=0, nx=nx, nstep=T, srci=si, srcj=sj, srcv=srcv, rcvi=ri, rcvj=rj)
    plan = ads.AcousticPlan(nx, NY, h, h, dt, [shot] * rep, npml=npml, vp_ref=vref,
                            precision="f32", variant=variant, ckpt_every=25)
    assert min(plan.rows) > 1  # (not the one-thread-per-cell kernels)

    def rel(x, y):
        return np.linalg.norm(x - y) / np.linalg.norm(y)

    vt = torch.as_tensor(vp, dtype=torch.float64, device=cuda)
    got = plan.split_traces(plan.forward(vt))
    assert rel(got[0].double().cpu().numpy(), tr) <= 1e-5
    o = torch.as_tensor(obs, device=cuda)
    l, g = plan.gradient(vt, plan.pack([o] * rep))
    torch.cuda.synchronize()
    assert abs(float(l) - rep * loss) <= 1e-4 * rep * loss
    g = g.cpu().numpy().reshape(nx + 2, NY + 2) / rep
    grad = np.asarray(grad).reshape(nx + 2, NY + 2)
    assert rel(g, grad) <= 1e-4
    cols = slice(edge - 8, edge + 1)  # the columns that were cut off
    assert rel(g[:, cols], grad[:, cols]) <= 1e-4
    plan.close()

"""Coordinates far off the grid, up to the infinite ones: the geometry never calls such a point
valid (on the host), and the 2-D, slow-Z and BOX routines grid and degrid the others as if it were
not there, its WT negated like any point's outside the grid."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import small_obs

HERE = os.path.dirname(os.path.abspath(__file__))
FAR = [np.inf, -np.inf, 1e30, -1e30, 3e9, -3e9, 5e10]


def test_far_cells_are_not_valid(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "cell_limits")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fwrapv", "-I",
                    os.path.join(HERE, "..", "sde_gb300", "csrc"), os.path.join(HERE, "cell_limits.cpp"), "-o", exe, "-lm"],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    points, bad = (int(x) for x in out.stdout.split())
    assert points > 5000 and bad == 0, out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [(0.0, 0.0), (30.0, -20.0)])
def test_far_points_in_a_plan(gpu_ctx, shift):
    from sde_gb300.imaging import Geom, Plan
    ctx, torch = gpu_ctx, gpu_ctx.torch
    g = Geom(128, 4.0, vdec=50.0, shift=shift)
    rng = np.random.default_rng(1)
    n, far = 3000, len(FAR) ** 2
    u = (rng.uniform(-0.9, 0.9, n) * g.nu / float(g.uscale)).astype(np.float32)
    v = (rng.uniform(-0.45, 0.45, n) * g.nv / float(g.vscale)).astype(np.float32)
    vis = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    at = np.arange(10, 10 + 5 * far, 5)
    fu, fv = u.copy(), v.copy()
    for i, (a, b) in enumerate((a, b) for a in FAR for b in [0.0] + FAR[1:]):
        fu[at[i]], fv[at[i]] = (a, b) if i % 2 else (b, a)
    model = torch.zeros((g.nv, g.pitch), dtype=torch.complex64, device=ctx.device)
    model[:, :g.nu] = ctx.tensor((rng.standard_normal((g.nv, g.nu)) + 1j).astype(np.complex64))
    keep = np.ones(n, bool)
    keep[at] = False
    got = []
    for uu, vv, wt in ((fu, fv, np.ones(n, np.float32)), (u, v, keep.astype(np.float32))):  # far, or without weight
        t = [ctx.tensor(a, torch.float32) for a in (uu, vv, np.zeros(n))] + [ctx.tensor(vis), ctx.tensor(wt)]
        p = Plan(ctx, g, *t)
        grid = ctx.grid_buffer(g)
        p.grid(grid)
        p.degrid_residual(model)
        res = p.residual(ctx.zeros(n, torch.complex64))
        out, ow = ctx.zeros(n, torch.complex64), ctx.tensor(wt)
        p.degrid(model, out, ow)
        ctx.sync()
        got.append([a.cpu().numpy() for a in (grid, res, out, ow)])
        p.close()
    a, b = got
    assert np.abs(a[0] - b[0]).max() <= 1e-5 * np.abs(b[0]).max()
    assert np.array_equal(a[1][keep], b[1][keep]) and np.array_equal(a[2][keep], b[2][keep])
    assert (a[3][keep] == b[3][keep]).all()
    assert (a[3][at] == -1.0).all() and (a[2][at] == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("far", FAR)
def test_far_points_box_and_slow_z(gpu_ctx, orc, far):
    from sde_gb300 import _abi
    from test_box import _grdqh2d
    from test_slowz import CELLZ, REFZ, NZ, _grddeh23, _grdh23d
    L = _abi.lib()
    o = small_obs(imsize=64, cell=8.0, ntime=4, jitter=True)
    p = orc.params(64, 8.0, fov=1.0, rmode="NONE", vdec=o["vdec"], shift=o["shift"])
    g = orc.geom(p)
    cf, _, _ = orc.grdcf()
    at = np.array([5, 50, 500])
    f = dict(o, u=o["u"].copy(), v=o["v"].copy(), wt=o["wt"].copy())
    f["u"][at[:2]] = far
    f["v"][at[1:]] = far
    off = dict(o, wt=o["wt"].copy())
    off["wt"][at] = 0.0
    a, b = _grdqh2d(L, f, g)[0], _grdqh2d(L, off, g)[0]
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
    a, b = _grdh23d(L, f, g, cf)[0], _grdh23d(L, off, g, cf)[0]
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
    model, _, _ = orc.grdh23d(o["vis"], o["wt"], o["u"], o["v"], o["w"], g, cf, NZ, CELLZ, REFZ)
    va, wa, err = _grddeh23(L, f, g, cf, model)
    vb, wb, _ = _grddeh23(L, o, g, cf, model)
    keep = np.ones(len(va), bool)
    keep[at] = False
    assert err == 0 and np.array_equal(va[keep], vb[keep]) and np.array_equal(wa[keep], wb[keep])
    assert (va[at] == 0).all() and np.array_equal(wa[at], -o["wt"][at])

"""FFT row and column passes at the lengths whose single launches take the narrow CTA shape
(64..2048 points a side with fewer than two CTAs per SM), against the oracle's FFTR2D: images
narrower and shorter than the transform, the last CTA with one row, a grid pitch whose last
column is padding.  2e-6 of the largest value, as the other FFT comparisons here: at most four
radix passes of a few roundings each."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,fnu,nv", [
    (64, 64, 64, 64), (37, 41, 64, 128),          # 16 rows a CTA; 8 and 16 columns
    (128, 127, 128, 128), (101, 9, 128, 32),       # 8 rows
    (251, 257, 256, 512), (256, 253, 256, 256),   # 4 rows; 2 and 4 columns
    (500, 301, 512, 512), (511, 130, 512, 1024),  # 2 rows
    (1024, 513, 1024, 1024), (999, 75, 1024, 256),    # 1 row
    (1023, 61, 2048, 128), (2047, 35, 2048, 64), (4093, 5, 4096, 32),  # rows longer than 512
])
def test_narrow_shapes(gpu_ctx, orc, nx, ny, fnu, nv):
    ctx = gpu_ctx
    rng = np.random.default_rng(nx * 7 + ny)
    nu = fnu // 2 + 1
    pitch = (nu + 3) & ~3

    class G:
        pass
    g = G()
    g.pitch, g.nx, g.ny, g.fnu, g.nv = pitch, nx, ny, fnu, nv
    X = (rng.standard_normal((nv, nu)) + 1j * rng.standard_normal((nv, nu))).astype(np.complex64)
    ref_img, _ = orc.fftr2d(nx, ny, fnu, nv, -1, xarray=X)
    Xp = np.zeros((nv, pitch), np.complex64)
    Xp[:, :nu] = X
    grid = ctx.tensor(Xp)
    img = ctx.empty((ny, nx), ctx.torch.float32)
    ctx.image_from_grid(g, grid, img, correct=False)
    assert rel_err(img.cpu().numpy(), ref_img) < 2e-6
    im = rng.standard_normal((ny, nx)).astype(np.float32)
    _, refX = orc.fftr2d(nx, ny, fnu, nv, +1, rarray=im)
    back = ctx.zeros((nv, pitch), ctx.torch.complex64)
    ctx.grid_from_image(g, ctx.tensor(im), back, correct=False)
    assert rel_err(back.cpu().numpy()[:, :nu], refX) < 2e-6


# IMGDOUBL's padding folded into the transform: the grid of the padded image, at margins that
# are even and odd, with images of one row or column, and where whole 256-row boxes of the
# column pass's input hold no image row (2048 and 4096 rows)
@pytest.mark.parametrize("nx,ny,lsx,lsy,px,py", [(33, 30, 15, 17, 64, 64), (1, 7, 5, 0, 16, 16), (100, 1, 14, 127, 128, 128),
                                                 (501, 499, 262, 263, 1024, 1024), (300, 900, 0, 1148, 2048, 2048),
                                                 (750, 700, 649, 675, 2048, 2048), (1499, 1499, 1298, 1298, 4096, 4096),
                                                 (2048, 100, 1024, 2000, 4096, 4096)])
@pytest.mark.parametrize("correct", [False, True])
def test_grid_of_padded_image(gpu_ctx, nx, ny, lsx, lsy, px, py, correct):
    """Equal to padding first: the same operations on the same numbers (zeros of either sign)."""
    from sde_gb300._abi import check, lib
    from sde_gb300.imaging import _ptr
    ctx, torch = gpu_ctx, gpu_ctx.torch
    rng = np.random.default_rng(nx + ny)
    im = ctx.tensor(rng.standard_normal((ny, nx)).astype(np.float32))
    pad = ctx.zeros((py, px), torch.float32)
    pad[lsy:lsy + ny, lsx:lsx + nx] = im
    pitch = (px // 2 + 1 + 3) & ~3
    want = ctx.zeros((py, pitch), torch.complex64)
    got = torch.full_like(want, float("nan"))
    check(lib().sde_grid_from_image(ctx.h, _ptr(pad), px, py, px, py, int(correct), _ptr(want), pitch), "image")
    check(lib().sde_grid_from_padded(ctx.h, _ptr(im), nx, ny, lsx, lsy, px, py, px, py, int(correct), _ptr(got), pitch),
          "padded")
    nu = px // 2 + 1
    assert torch.equal(torch.view_as_real(got[:, :nu]), torch.view_as_real(want[:, :nu]))


def test_padded_image_must_lie_inside(gpu_ctx):
    from sde_gb300._abi import lib
    from sde_gb300.imaging import _ptr
    ctx, torch = gpu_ctx, gpu_ctx.torch
    im, g = ctx.zeros((8, 8), torch.float32), ctx.zeros((32, 20), torch.complex64)
    for nx, ny, lsx, lsy in ((8, 8, -1, 0), (8, 8, 25, 0), (8, 8, 0, 25), (0, 8, 0, 0)):
        assert lib().sde_grid_from_padded(ctx.h, _ptr(im), nx, ny, lsx, lsy, 32, 32, 32, 32, 0, _ptr(g), 20) == 1


# the row-pair kernel: four pixels a thread, image widths that are any multiple of 4 (the first
# pixel's place in the transform wraps or not), odd row counts, and 512-long half-rows in a batch
@pytest.mark.parametrize("nx,ny,n", [(4, 3, 2048), (2044, 2047, 2048), (1028, 9, 2048), (4096, 5, 4096), (2052, 33, 4096),
                                     (8188, 7, 8192), (1020, 1024, 1024)])
def test_row_pairs(gpu_ctx, orc, nx, ny, n):
    ctx = gpu_ctx
    rng = np.random.default_rng(nx + ny)
    nv, nu = 64 if ny <= 64 else n, n // 2 + 1
    pitch = (nu + 3) & ~3

    class G:
        pass
    g = G()
    g.pitch, g.nx, g.ny, g.fnu, g.nv = pitch, nx, ny, n, nv
    X = (rng.standard_normal((nv, nu)) + 1j * rng.standard_normal((nv, nu))).astype(np.complex64)
    ref, _ = orc.fftr2d(nx, ny, n, nv, -1, xarray=X)
    Xp = np.zeros((nv, pitch), np.complex64)
    Xp[:, :nu] = X
    img = ctx.empty((ny, nx), ctx.torch.float32)
    scale = ctx.tensor(np.array([4.0], np.float32))
    ctx.image_from_grid(g, ctx.tensor(Xp), img, correct=False, scale_dev=scale)
    assert rel_err(img.cpu().numpy(), ref * np.float32(0.25)) < 2e-6


# the finalize inside the register column passes: every length, images narrower than the grid
@pytest.mark.parametrize("imsize,cell", [(64, 8.0), (100, 5.0), (500, 1.0), (1024, 0.5)])
def test_finalize_in_short_columns(gpu_ctx, obs_small, imsize, cell):
    """sde_plan_image against sde_plan_grid + sde_image_from_grid: the image bars of the two
    gridding passes' FP32 rounding (1e-5 of the peak in the CLEAN window, 5e-3 at the corners)."""
    from sde_gb300.imaging import Geom, Plan
    ctx, torch, o = gpu_ctx, gpu_ctx.torch, obs_small
    g = Geom(imsize, cell, vdec=o["vdec"])
    t = {k: ctx.tensor(o[k], None) for k in ("u", "v", "w", "wt", "vis")}
    plan = Plan(ctx, g, t["u"], t["v"], t["w"], t["vis"], t["wt"])
    for psf in (True, False):
        ga, gb, ia, ib = ctx.grid_buffer(g), ctx.grid_buffer(g), ctx.image_buffer(g), ctx.image_buffer(g)
        plan.grid(ga, psf=psf)
        ctx.image_from_grid(g, ga, ia)
        plan.image(ib, gb, psf=psf)
        ctx.sync()
        a, b = ia.cpu().numpy(), ib.cpu().numpy()
        w = slice(imsize // 4, imsize // 4 + imsize // 2 - 1)
        pk = np.abs(a).max()
        assert np.abs(a - b)[w, w].max() / pk < 1e-5
        assert np.abs(a - b).max() / pk < 5e-3
        assert float((ga - gb)[:, :g.nu].abs().max()) / float(ga.abs().max()) < 1e-5
    plan.close()

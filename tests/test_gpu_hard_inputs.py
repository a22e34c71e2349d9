"""Inputs at the limits of the CLEAN, transform and plan kernels: NaN and infinite pixels,
bulk-copied image rows with odd margins, work items of more chunks than are put in order, and
Clark lists whose pixels take several components in the one major cycle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# each Hogbom kernel: one cluster (four sizes), the chip's registers, the grid-wide one
@pytest.mark.parametrize("nx,ny", [(60, 50), (150, 140), (300, 300), (500, 500), (700, 500), (200, 1400)])
@pytest.mark.parametrize("kind", ["nan", "inf", "all_nan", "nan_psf"])
def test_hogbom_non_finite(gpu_ctx, orc, nx, ny, kind):
    """PIXISAMA's comparison never takes a NaN (pix/pixisama.f); the rest is PIX2DRCL's arithmetic,
    bit for bit (NaN for NaN)."""
    ctx = gpu_ctx
    rng = np.random.default_rng(nx + ny)
    psf = (0.1 * rng.standard_normal((2 * ny + 1, 2 * nx + 1))).astype(np.float32)
    psf[ny, nx] = 1.0
    drt = rng.standard_normal((ny, nx)).astype(np.float32)
    if kind == "nan":
        drt.reshape(-1)[rng.choice(nx * ny, 40, replace=False)] = np.nan
        drt[0, 0] = drt[-1, -1] = np.nan
    elif kind == "inf":
        drt[ny // 3, nx // 2] = -np.inf
    elif kind == "all_nan":
        drt[:] = np.nan
    else:
        psf[ny - 3, nx + 2] = np.nan
    niter = 6
    r = ctx.hogbom(ctx.tensor(drt), ctx.tensor(psf), niter, 0.3)
    if kind == "all_nan":  # nothing to subtract
        assert r["ansub"] == 0 and not r["cln"].any()
        return
    o = orc.pix2drcl(drt, psf, np.ones_like(drt), 0.3, niter)
    assert r["ansub"] == o["ansub"]
    for k in ("cx", "cy", "cflux", "cln", "res"):
        assert np.array_equal(r[k].cpu().numpy(), o[k], equal_nan=k not in ("cx", "cy")), k


@pytest.mark.parametrize("nx,ny,lsx,lsy,p", [(4000, 40, 33, 7, 4096), (4, 3, 4091, 1, 4096), (4096, 17, 0, 3, 4096),
                                             (1000, 9, 1547, 5, 8192)])
@pytest.mark.parametrize("correct", [False, True])
def test_bulk_rows_with_odd_margins(gpu_ctx, nx, ny, lsx, lsy, p, correct):
    """Equal to padding first: the same operations on the same numbers."""
    from sde_gb300._abi import check, lib
    from sde_gb300.imaging import _ptr
    ctx, torch = gpu_ctx, gpu_ctx.torch
    py = 64
    im = ctx.tensor(np.random.default_rng(nx).standard_normal((ny, nx)).astype(np.float32))
    pad = ctx.zeros((py, p), torch.float32)
    pad[lsy:lsy + ny, lsx:lsx + nx] = im
    nu = p // 2 + 1
    pitch = (nu + 3) & ~3
    want, got = (ctx.zeros((py, pitch), torch.complex64) for _ in range(2))
    check(lib().sde_grid_from_image(ctx.h, _ptr(pad), p, py, p, py, int(correct), _ptr(want), pitch), "image")
    check(lib().sde_grid_from_padded(ctx.h, _ptr(im), nx, ny, lsx, lsy, p, py, p, py, int(correct), _ptr(got), pitch),
          "padded")
    assert torch.equal(torch.view_as_real(got[:, :nu]), torch.view_as_real(want[:, :nu]))


# chunks of 4 visibilities: 2048 cell pairs (of two chunks each: 4096), and one chunk over
@pytest.mark.parametrize("per,extra", [(8, 0), (8, 1), (20, 0)])
def test_items_of_many_chunks(gpu_ctx, per, extra):
    """The image bar of two gridding passes' FP32 rounding, 1e-5 of the peak in the CLEAN window."""
    from sde_gb300.imaging import Geom, Plan
    ctx, torch = gpu_ctx, gpu_ctx.torch
    g = Geom(256, 1.0, vdec=40.0)
    cu, cv = np.meshgrid(np.arange(64, 128), np.arange(64, 128))  # the cells of one tile (0-based)
    cell = np.repeat(np.arange(cu.size), per // 2)
    cell = np.concatenate([cell, np.zeros(extra, int)])
    rng = np.random.default_rng(per)
    rng.shuffle(cell)
    u = ((cu.reshape(-1)[cell] + 1 - g.uorigin) / g.uscale).astype(np.float32)
    v = ((cv.reshape(-1)[cell] + 1 - g.vorigin) / g.vscale).astype(np.float32)
    n = len(u)
    vis = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    wt = rng.uniform(0.5, 1.5, n).astype(np.float32)
    t = [ctx.tensor(a, torch.float32) for a in (u, v, np.zeros(n))] + [ctx.tensor(vis), ctx.tensor(wt)]
    mgrid = ctx.grid_buffer(g)
    mgrid[:, :g.nu] = ctx.tensor((rng.standard_normal((g.nv, g.nu)) + 1j).astype(np.complex64))
    got = []
    for opts in (None, (65536, 4)):
        p = Plan(ctx, g, *t, opts=opts)
        im = ctx.image_buffer(g)
        p.image(im)
        p.degrid_residual(mgrid)
        res = p.residual(ctx.zeros(n, torch.complex64))
        ctx.sync()
        got.append((im.cpu().numpy(), res.cpu().numpy()))
        p.close()
    w = slice(64, 191)
    assert np.abs(got[0][0] - got[1][0])[w, w].max() / np.abs(got[0][0]).max() < 1e-5
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-5 * np.abs(got[0][1]).max()


@pytest.mark.parametrize("numcl,bp,niter", [(32768, 128, 40), (32768, 128, 150), (20000, 300, 120), (5000, 64, 60)])
def test_clark_component_sums(gpu_ctx, orc, numcl, bp, niter):
    """One major cycle, so the component image and the scalars are the oracle's too, bit for bit;
    a gain of 0.1 on a few bright points gives their pixels many components each."""
    from sde_gb300.imaging import clark
    ctx, n = gpu_ctx, 512
    rng = np.random.default_rng(numcl + bp)
    y, x = np.mgrid[0:n, 0:n]
    c = (n + 1) // 2 - 1
    r2 = (x - c) ** 2 + (y - c) ** 2
    psf = np.exp(-r2 / 18.0).astype(np.float32)
    dirty = (0.01 * rng.standard_normal((n, n))).astype(np.float32)
    for f, px, py in zip(rng.uniform(3.0, 5.0, 6), rng.integers(140, 370, 6), rng.integers(140, 370, 6)):
        dirty += np.float32(f) * np.roll(psf, (py - c, px - c), (0, 1))
    o = orc.clark(dirty, psf, niter=niter, gain=0.1, flux=0.0, numcl=numcl, bpatch=bp)
    g = clark(ctx, ctx.tensor(dirty), ctx.tensor(psf), niter=niter, gain=0.1, flux=0.0, numcl=numcl, bpatch=bp)
    a = o["trace"][0][1]
    assert o["ncycles"] == 1 and a == niter
    assert len(set(zip(o["cx"][:a].tolist(), o["cy"][:a].tolist()))) < a / 2
    assert g["ncycles"] == 1 and g["trace"][0][:2] == o["trace"][0][:2]
    for k in ("cl", "cx", "cy"):
        assert np.array_equal(g[k].cpu().numpy()[:a], o[k][:a]), k
    assert np.array_equal(g["comp"].cpu().numpy(), o["comp"])
    assert g["maxres"] == o["maxres"] and g["tflux"] == o["tflux"]

"""Direct transforms at the edges of their tiles (64 x 64 pixels; 64 visibilities by bands of 64,
96 or 128 rows; chunks of 32) and of the phase reduction, against exact phases in FP64: 1e-5 of
the peak, the repository's bar for both transforms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vis(n, seed, turns):
    rng = np.random.default_rng(seed)
    u, v = (rng.uniform(-turns, turns, n) * 3600.0 / 2.0 * 180.0 / np.pi for _ in range(2))  # 2 arcsec pixels
    vis = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    wt = rng.uniform(0.5, 1.5, n)
    wt[rng.uniform(size=n) < 0.1] = -1.0
    wt[0] = 1.0
    return [a.astype(np.float32) for a in (u, v)] + [vis.astype(np.complex64), wt.astype(np.float32)]


# turns per pixel up to half (the sampling limit), and past a whole turn
@pytest.mark.parametrize("n,nx,ny,rx,ry,turns", [
    (1, 1, 1, 1.0, 1.0, 0.5), (31, 63, 65, 32.0, 33.0, 0.5), (32, 64, 64, 32.5, 32.0, 0.5), (33, 65, 96, 1.0, 48.5, 0.5),
    (63, 2, 97, 1.5, 40.0, 0.5), (64, 128, 128, 64.0, 64.0, 0.5), (65, 33, 129, 17.0, 65.0, 0.5),
    (2100, 70, 50, 35.0, 25.0, 0.5), (500, 40, 30, 20.5, 15.0, 7.0)])
def test_edges(gpu_ctx, orc, n, nx, ny, rx, ry, turns):
    from sde_gb300.imaging import dft_image, dft_vis
    ctx = gpu_ctx
    u, v, vis, wt = _vis(n, n + nx, turns)
    d = 2.0 / 3600.0
    t = [ctx.tensor(a) for a in (u, v, vis, wt)]
    d64, p64, rc = orc.visdft2d(vis, wt, u, v, nx, ny, rx, -d, ry, d, fp64=True)
    assert rc == 0
    both = dft_image(ctx, *t, nx, ny, rx, -d, ry, d)
    one = dft_image(ctx, *t, nx, ny, rx, -d, ry, d, psf=False)
    two = dft_image(ctx, *t, nx, ny, rx, -d, ry, d, dirty=False)
    ctx.sync()
    for a in (both["dirty"], one["dirty"]):
        assert np.abs(a.cpu().numpy() - d64).max() <= 1e-5 * np.abs(d64).max()
    for a in (both["psf"], two["psf"]):
        assert np.abs(a.cpu().numpy() - p64).max() <= 1e-5
    image = np.random.default_rng(n).standard_normal((ny, nx)).astype(np.float32)
    old = np.full(n, 3 - 2j, np.complex64)
    got = dft_vis(ctx, ctx.tensor(image), rx, -d, ry, d, t[0], t[1], t[3], ctx.tensor(old))
    ctx.sync()
    v64 = orc.imgdft2d(image, rx, -d, ry, d, wt, u, v, vis_in=old, fp64=True)
    g = got.cpu().numpy()
    assert np.array_equal(g[wt <= 0], old[wt <= 0])
    assert np.abs(g - v64)[wt > 0].max() <= 1e-5 * np.abs(v64[wt > 0]).max()

"""Direct transforms about a reference pixel at any place, not only on or halfway between pixels,
for baselines within and beyond the sampling limit, against exact phases in FP64: 1e-5 of the
peak, the repository's bar for both transforms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turns", [0.5, 1.3, 7.0, 60.0])
@pytest.mark.parametrize("rx,ry", [(20.3, 15.0), (20.0, 15.25), (-3.7, 40.125), (20.5, 15.0), (1000.75, -8191.9)])
def test_reference_pixel(gpu_ctx, orc, rx, ry, turns):
    from sde_gb300.imaging import dft_image, dft_vis
    ctx, n, nx, ny, d = gpu_ctx, 300, 40, 30, 2.0 / 3600.0
    rng = np.random.default_rng(int(turns * 10))
    u, v = ((rng.uniform(-turns, turns, n) / d * 180.0 / np.pi).astype(np.float32) for _ in range(2))
    vis = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    wt = rng.uniform(0.5, 1.5, n).astype(np.float32)
    t = [ctx.tensor(a) for a in (u, v, vis, wt)]
    got = dft_image(ctx, *t, nx, ny, rx, -d, ry, d)
    d64, p64, rc = orc.visdft2d(vis, wt, u, v, nx, ny, rx, -d, ry, d, fp64=True)
    assert rc == 0
    assert np.abs(got["dirty"].cpu().numpy() - d64).max() <= 1e-5 * np.abs(d64).max()
    assert np.abs(got["psf"].cpu().numpy() - p64).max() <= 1e-5 * np.abs(p64).max()
    image = rng.standard_normal((ny, nx)).astype(np.float32)
    out = dft_vis(ctx, ctx.tensor(image), rx, -d, ry, d, t[0], t[1], t[3], ctx.zeros(n, ctx.torch.complex64))
    v64 = orc.imgdft2d(image, rx, -d, ry, d, wt, u, v, fp64=True)
    assert np.abs(out.cpu().numpy() - v64).max() <= 1e-5 * np.abs(v64).max()

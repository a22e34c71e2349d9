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

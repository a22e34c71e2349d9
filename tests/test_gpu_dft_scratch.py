"""IMGDFT2D on a tall image: the scratch of its bands is bounded whatever the number of
visibilities (256 MB, and an eighth of slack), which go through in slices with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_bands_in_slices(gpu_ctx, orc):
    from sde_gb300.imaging import Context, dft_vis
    ctx = Context(0)
    torch, ny, nx, n, d = ctx.torch, 8192, 3, 1200000, 2.0 / 3600.0
    rng = np.random.default_rng(3)
    u, v = (rng.uniform(-0.5, 0.5, n).astype(np.float32) / np.float32(d) * np.float32(180.0 / np.pi) for _ in range(2))
    wt = rng.uniform(0.5, 1.5, n).astype(np.float32)
    wt[::97] = -1.0
    image = rng.standard_normal((ny, nx)).astype(np.float32)
    t = [ctx.tensor(a) for a in (u, v, wt)]
    old = ctx.tensor(np.full(n, 3 - 2j, np.complex64))
    before = ctx_bytes(ctx)
    got = dft_vis(ctx, ctx.tensor(image), 2.0, -d, 4096.5, d, t[0], t[1], t[2], old)
    ctx.sync()
    assert ctx_bytes(ctx) - before < 9 / 8 * ((256 << 20) + 48 * n) + 4096  # bands, and the records
    got = got.cpu().numpy()
    assert np.array_equal(got[wt <= 0], np.full((wt <= 0).sum(), 3 - 2j, np.complex64))
    # where a slice of 256 MB of 64 bands of 128 rows ends, and elsewhere
    edge = (256 << 20) // (8 * 64)
    pick = np.unique(np.concatenate([np.arange(4), edge + np.arange(-3, 4), 2 * edge + np.arange(-3, 4), [n - 2, n - 1],
                                     rng.integers(0, n, 200)]))
    pick = pick[wt[pick] > 0]
    ref = orc.imgdft2d(image, 2.0, -d, 4096.5, d, wt[pick], u[pick], v[pick], fp64=True)
    assert np.abs(got[pick] - ref).max() <= 1e-5 * np.abs(ref).max()
    ctx.close()


def ctx_bytes(ctx):
    from sde_gb300._abi import lib
    return lib().sde_ctx_bytes_in_use(ctx.h)

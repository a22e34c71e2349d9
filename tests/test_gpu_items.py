"""Launch lists: a plan's images and residuals, and a batch's images, do not depend on whether
an item's rounds of chunks are dealt out to several teams or its visibilities are cut into
small items that one team takes whole (the repository's image bar: 1e-5 of the peak inside the
CLEAN window; only the order of FP32 sums differs)."""
import numpy as np
import pytest

from conftest import small_obs

pytestmark = pytest.mark.gpu


def _tensors(ctx, o):
    torch = ctx.torch
    t = {k: ctx.tensor(o[k], torch.float32) for k in ("u", "v", "w", "wt")}
    t["vis"] = ctx.tensor(np.asarray(o["vis"], np.complex64).view(np.float32), torch.float32)
    return t


def _close(a, b):
    n = a.shape[0]
    w = slice(n // 4, n // 4 + n // 2 - 1)
    assert np.abs(a - b)[w, w].max() / np.abs(b).max() < 1e-5


# ntime * 351 visibilities: one round, a ragged few, either side of the step from 256 to 512
# visibilities an entry (2^18), larger
@pytest.mark.parametrize("ntime", [1, 7, 746, 747, 3000])
def test_parts_equal_small_items(gpu_ctx, ntime):
    from sde_gb300.imaging import Geom, Plan
    ctx = gpu_ctx
    o = small_obs(imsize=256, cell=2.0, ntime=ntime, jitter=True)
    g = Geom(256, 2.0, vdec=40.0)
    t = _tensors(ctx, o)
    model = ctx.zeros((256, 256), ctx.torch.float32)
    model[100, 140] = 0.7
    mgrid = ctx.grid_buffer(g)
    ctx.grid_from_image(g, model, mgrid)
    got = []
    for opts in (None, (256, 64)):
        p = Plan(ctx, g, t["u"], t["v"], t["w"], t["vis"], t["wt"], opts=opts)
        im = ctx.image_buffer(g)
        p.image(im)
        p.degrid_residual(mgrid)
        res = p.residual(ctx.empty(len(o["u"]), ctx.torch.complex64))
        ctx.sync()
        got.append((im.cpu().numpy(), res.cpu().numpy()))
        p.close()
    _close(got[0][0], got[1][0])
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-5 * np.abs(got[1][1]).max()


@pytest.mark.parametrize("ntime", [100, 800, 3100])
def test_batch_parts_equal_small_items(gpu_ctx, ntime):
    from sde_gb300.mosaic import Mosaic
    obs = [small_obs(imsize=256, cell=2.0, ntime=nt, seed=7 + i) for i, nt in enumerate((ntime, 3, 40))]
    pts = [dict(o, imsize=256, l0=0.0, m0=1e-3 * i, pb_fwhm_rad=0.01) for i, o in enumerate(obs)]
    got = []
    for opts in (None, (256, 64)):
        m = Mosaic(gpu_ctx, pts, 2.0, opts=opts, mosaic=False)
        m.dirty(graph=False)
        m.dirty(graph=True)
        got.append([m.read(i) for i in range(m.n)])
        m.close()
    for a, b in zip(*got):
        _close(a, b)

"""Hogbom windows that one thread-block cluster holds (up to 262144 pixels): the component
list, residual and component image are PIX2DRCL's, bit for bit, at the sizes where the pixels
per thread change, on ragged and one-pixel windows, with a box, for every stop rule, and where
the PSF does not cover every shift (the grid-wide kernel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(nx, ny, pnx, pny, seed):
    rng = np.random.default_rng(seed)
    psf = (0.1 * rng.standard_normal((pny, pnx))).astype(np.float32)
    psf[pny // 2, pnx // 2] = 1.0
    drt = rng.standard_normal((ny, nx)).astype(np.float32)
    return drt, psf


def _compare(ctx, orc, drt, psf, niter, gain=0.1, flux=0.0, box=None, bsub=1, tflux=0.0):
    torch = ctx.torch
    r = ctx.hogbom(ctx.tensor(drt), ctx.tensor(psf), niter, gain, flux=flux, bsub=bsub, tflux=tflux,
                   box=None if box is None else ctx.tensor(box))
    one = np.ones_like(drt) if box is None else box
    o = orc.pix2drcl(drt, psf, one, gain, niter, bsub=bsub, flux=flux, tflux=tflux)
    assert r["ansub"] == o["ansub"]
    for k in ("cx", "cy", "cflux", "cln", "res"):
        assert np.array_equal(r[k].cpu().numpy(), o[k]), k
    assert np.float32(r["maxres"]) == np.float32(o["maxres"])
    assert np.float32(r["tflux"]) == np.float32(o["tflux"])
    assert torch.isfinite(r["res"]).all()


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 40), (7, 5), (63, 65), (128, 128), (129, 127), (255, 255), (256, 257),
                                   (361, 361), (363, 362), (512, 512), (513, 512)])
def test_window_sizes(gpu_ctx, orc, nx, ny):
    drt, psf = _case(nx, ny, 2 * nx + 1, 2 * ny + 1, nx * 1000 + ny)
    _compare(gpu_ctx, orc, drt, psf, 12)


@pytest.mark.parametrize("kw", [dict(niter=-40), dict(niter=40, flux=2.0), dict(niter=300, gain=0.3, bsub=4, tflux=1.5),
                                dict(niter=0), dict(niter=600, gain=0.05)])
def test_stop_rules_and_long_runs(gpu_ctx, orc, kw):
    drt, psf = _case(61, 47, 128, 100, 3)
    _compare(gpu_ctx, orc, drt, psf, **kw)


def test_box_and_uncovered_psf(gpu_ctx, orc):
    drt, psf = _case(90, 70, 200, 150, 5)
    box = np.zeros((70, 90), np.float32)
    box[20:50, 30:80] = 1.0
    _compare(gpu_ctx, orc, drt, psf, 30, box=box)
    drt, psf = _case(90, 70, 96, 80, 6)  # smaller than twice the window
    _compare(gpu_ctx, orc, drt, psf, 30)


def test_zero_residual(gpu_ctx, orc):
    drt, psf = _case(40, 30, 81, 61, 7)
    _compare(gpu_ctx, orc, np.zeros_like(drt), psf, 10)


# windows above the cluster's, in the registers of one CTA per SM: few and many pixels a thread,
# rows of exactly a thread's step and one less (the general kernel), a narrow and a wide window,
# the last CTA short or empty, the largest window that fits (152 x 256 x 108 pixels) and one over
@pytest.mark.parametrize("nx,ny,box", [(513, 513, False), (256, 1030, True), (255, 1040, False), (700, 391, True),
                                       (5000, 53, False), (1023, 1023, True), (2047, 2047, False), (1152, 3648, False),
                                       (1153, 3648, True)])
def test_windows_in_registers(gpu_ctx, orc, nx, ny, box):
    drt, psf = _case(nx, ny, 2 * nx + 3, 2 * ny, nx + ny)
    b = None
    if box:
        b = (np.random.default_rng(ny).random((ny, nx)) > 0.3).astype(np.float32)
    _compare(gpu_ctx, orc, drt, psf, 9, gain=0.4, box=b, bsub=2)


def test_register_window_stop_rules(gpu_ctx, orc):
    drt, psf = _case(600, 500, 1201, 1001, 11)
    drt[3, 5] = -9.0
    _compare(gpu_ctx, orc, drt, psf, -40)         # a negative maximum stops at once
    _compare(gpu_ctx, orc, drt, psf, 40, flux=4.0)
    _compare(gpu_ctx, orc, drt, psf, 0)
    _compare(gpu_ctx, orc, np.zeros_like(drt), psf, 5)

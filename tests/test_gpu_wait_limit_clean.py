"""CLEAN minor cycles whose waits for the other blocks' maxima run out: SDE_ETIMEDOUT or the whole,
right result, never a hang, and the context works as before.  Limits of a few polls make some
warps of a block run out and not others, in the first round, in the last and between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITS = [0, 1, 2, 4, 8, 16, 64]


def _limited(ctx, limit, f):
    """f() under the limit: its result, or None when it timed out."""
    from sde_gb300 import _abi
    L = _abi.lib()
    L.sde_ctx_set_wait_limit(ctx.h, limit)
    try:
        r = f()
    except RuntimeError:
        assert "timed out" in _abi.last_error()
        r = None
    finally:
        L.sde_ctx_set_wait_limit(ctx.h, -1)
    L.sde_ctx_sync(ctx.h)  # (reports the time-out once more)
    return r


# one cluster (its four sizes), then the chip's registers; runs past the cluster kernel's ring of
# 256 components, runs that end with it, and runs of no component at all
@pytest.mark.parametrize("nx,ny", [(60, 50), (150, 140), (300, 300), (500, 500), (700, 500)])
@pytest.mark.parametrize("niter", [0, 1, 256, 300])
def test_hogbom(gpu_ctx, orc, nx, ny, niter):
    ctx = gpu_ctx
    rng = np.random.default_rng(nx + niter)
    psf = (0.1 * rng.standard_normal((2 * ny + 1, 2 * nx + 1))).astype(np.float32)
    psf[ny, nx] = 1.0
    drt = rng.standard_normal((ny, nx)).astype(np.float32)
    dev = ctx.tensor(drt), ctx.tensor(psf)
    o = orc.pix2drcl(drt, psf, np.ones_like(drt), 0.05, niter)

    def same(r):
        assert r["ansub"] == o["ansub"]
        for k in ("cx", "cy", "cflux", "cln", "res"):
            a = r[k].cpu().numpy()
            assert np.array_equal(a[:niter] if a.ndim == 1 else a, o[k][:niter] if a.ndim == 1 else o[k]), k

    for limit in LIMITS:
        r = _limited(ctx, limit, lambda: ctx.hogbom(*dev, niter, 0.05))
        assert limit > 0 or r is None
        if r is not None:
            same(r)
        same(ctx.hogbom(*dev, niter, 0.05))


@pytest.mark.parametrize("niter", [1, 40, 300])
def test_clark(gpu_ctx, niter):
    from sde_gb300.imaging import clark
    ctx, n = gpu_ctx, 512
    rng = np.random.default_rng(niter)
    y, x = np.mgrid[0:n, 0:n]
    c = (n + 1) // 2 - 1
    psf = np.exp(-((x - c) ** 2 + (y - c) ** 2) / 18.0).astype(np.float32)
    dirty = (0.05 * rng.standard_normal((n, n))).astype(np.float32)
    dev = ctx.tensor(dirty), ctx.tensor(psf)
    run = lambda: clark(ctx, *dev, niter=niter, gain=0.1)  # noqa: E731
    want = run()
    for limit in LIMITS:
        r = _limited(ctx, limit, run)
        assert limit > 0 or r is None
        for got in ([r] if r is not None else []) + [run()]:
            for k in ("comp", "resid", "cl", "cx", "cy"):
                assert ctx.torch.equal(got[k], want[k]), k

"""SUMWT of weights whose partial sums leave the REALs: the reference's sum is DOUBLE
(grd/grdruw2d.f:132-159), within 1e-12 of a 64-bit sum here (any order of DOUBLE additions of a few
thousand positive terms), and infinite only for an infinite weight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 5000, 70001])
@pytest.mark.parametrize("scale", [1.0, 2e37, 3e38])
def test_sumwt(gpu_ctx, n, scale):
    from sde_gb300.imaging import Geom
    ctx, g = gpu_ctx, Geom(512, 1.0, vdec=40.0)
    rng = np.random.default_rng(n)
    u, v = (rng.uniform(-200, 200, n).astype(np.float32) / np.float32(s) for s in (g.wuscale, g.wvscale))
    wt = (scale * rng.uniform(0.5, 1.0, n)).astype(np.float32)
    t = [ctx.tensor(a, ctx.torch.float32) for a in (u, v, np.zeros(n), wt)]
    st = ctx.weights(g, *t, rmode="UNIFORM", newwt=ctx.zeros(n, ctx.torch.float32))
    assert st.ndrop == 0
    assert abs(st.sumwt / wt.astype(np.float64).sum() - 1.0) < 1e-12
    wt[n // 3] = np.inf
    t[3] = ctx.tensor(wt, ctx.torch.float32)
    assert ctx.weights(g, *t, rmode="UNIFORM", newwt=ctx.zeros(n, ctx.torch.float32)).sumwt == np.inf

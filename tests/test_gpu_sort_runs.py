"""Weight-density counts over the sizes where the sort's tiles, the runs' kernels and the
parallel form of the sequential FP32 sum change: every GWT cell and weight is the oracle's
sequential sum, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(ctx, orc, g, u, v, wt):
    torch = ctx.torch
    w = np.zeros_like(u)
    t = [ctx.tensor(a, torch.float32) for a in (u, v, w, wt)]
    gwt = ctx.empty((g.nv, g.nu), torch.float32)
    new = ctx.tensor(wt, torch.float32)
    ctx.weights(g, t[0], t[1], t[2], t[3], rmode="UNIFORM", gwt=gwt, newwt=new)
    ctx.sync()
    ref_new, ref_gwt, _ = orc.grduwt2d(wt, u, v, w, g.wuscale, g.wvscale, g.uorigin, g.vorigin, g.nu, g.nv,
                                       np.asarray(g.shift))
    assert np.array_equal(gwt.cpu().numpy().reshape(-1), np.asarray(ref_gwt).reshape(-1))
    got = new.cpu().numpy()
    assert np.array_equal(got[wt > 0], ref_new[wt > 0])  # (points with WT <= 0 are not written)
    assert np.array_equal(got[wt <= 0], wt[wt <= 0])


def _geom():
    from sde_gb300.imaging import Geom
    return Geom(64, 8.0, vdec=40.0)


# around one and two tiles of either size, and around the change of tile
@pytest.mark.parametrize("n", [1, 31, 2047, 2048, 2049, 4097, 1867775, 1867776, 1867777, 1880065])
def test_tile_edges(gpu_ctx, orc, n):
    g = _geom()
    rng = np.random.default_rng(n)
    u = (rng.uniform(-33, 33, n) / g.wuscale).astype(np.float32)
    v = (rng.uniform(-33, 33, n) / g.wvscale).astype(np.float32)
    wt = rng.uniform(0.1, 4.0, n).astype(np.float32)
    wt[rng.uniform(size=n) < 0.05] = -1.0
    _check(gpu_ctx, orc, g, u, v, wt)


# runs around the lengths that one thread sums (512) and one block of the parallel sum (512), and
# long ones; weights that round, that end on ties to even, that jump binades, that are tiny or
# huge beside the sum
@pytest.mark.parametrize("n", [511, 512, 513, 1023, 1024, 1025, 1537, 60000])
@pytest.mark.parametrize("kind", ["plain", "ties", "binades", "extreme"])
def test_long_runs(gpu_ctx, orc, n, kind):
    g = _geom()
    rng = np.random.default_rng(n)
    cell = rng.integers(0, 3, 3 * n)  # three long runs, interleaved in visibility order
    u = ((cell - 1) * 3.0 / g.wuscale).astype(np.float32)
    v = np.full(3 * n, 5.0 / g.wvscale, np.float32)
    wt = {"plain": lambda: rng.uniform(0.5, 1.5, 3 * n),
          "ties": lambda: rng.integers(1, 2000, 3 * n) + 0.5 * rng.integers(0, 2, 3 * n) + 4.0e6 * (np.arange(3 * n) < 8),
          "binades": lambda: 2.0 ** rng.integers(-12, 13, 3 * n),
          "extreme": lambda: 10.0 ** rng.uniform(-40, 30, 3 * n)}[kind]().astype(np.float32)
    _check(gpu_ctx, orc, g, u, v, wt)

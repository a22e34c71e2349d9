"""Device waits that give up: the sorts and scans of the weighting and of a plan end with
SDE_ETIMEDOUT (at once, or at the next sde_ctx_sync where the call does not wait), never with a
result, and the context works as before afterwards.  Small limits make the waits run out; what an
earlier, larger job left in the scratch is what a sort that gave up leaves in its place."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from sde_gb300.imaging import Context
    c = Context(0)
    yield c
    c.close()


def _job(ctx, imsize, n, seed):
    from sde_gb300.imaging import Geom
    g = Geom(imsize, 1.0, vdec=40.0)
    rng = np.random.default_rng(seed)
    u = (rng.uniform(-g.nu + 8, g.nu - 8, n) / g.wuscale).astype(np.float32)
    v = (rng.uniform(-g.nv / 2 + 8, g.nv / 2 - 8, n) / g.wvscale).astype(np.float32)
    vis = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    wt = rng.uniform(0.5, 1.5, n).astype(np.float32)
    return g, [ctx.tensor(a, ctx.torch.float32) for a in (u, v, np.zeros(n))] + [ctx.tensor(vis), ctx.tensor(wt)]


def _weights(ctx, g, t, stats):
    """(return code, new weights, GWT)"""
    from sde_gb300 import _abi
    from sde_gb300.imaging import _ptr
    n = t[4].numel()
    new, gwt = ctx.zeros(n, ctx.torch.float32), ctx.zeros((g.nv, g.nu), ctx.torch.float32)
    st = _abi.WStats()
    rc = _abi.lib().sde_weights(ctx.h, 0, (C.c_float * 3)(), 0.0, _ptr(t[4]), _ptr(t[0]), _ptr(t[1]), _ptr(t[2]), n,
                                float(g.wuscale), 0.0, float(g.wvscale), 0.0, g.uorigin, g.vorigin, g.nu, g.nv,
                                g.shift.ctypes.data_as(C.c_void_p), _ptr(new), _ptr(gwt),
                                C.byref(st) if stats else None)
    if not stats and rc == _abi.SDE_OK:
        rc = _abi.lib().sde_ctx_sync(ctx.h)
    return rc, new, gwt


def _plan(ctx, g, t):
    """(return code, chunk order of the plan as its residuals' grid)"""
    from sde_gb300 import _abi
    from sde_gb300.imaging import Plan
    try:
        p = Plan(ctx, g, t[0], t[1], t[2], t[3], t[4])
    except RuntimeError:
        return _abi.SDE_ETIMEDOUT if "timed out" in _abi.last_error() else -1, None
    grid = ctx.grid_buffer(g)
    p.grid(grid)
    ctx.sync()
    p.close()
    return _abi.SDE_OK, grid


# one tile of the sort and two of the scan over runs; a few and many tiles of either
@pytest.mark.parametrize("n", [2048, 5000, 40000, 2000000])
@pytest.mark.parametrize("limit", [0, 1, 2, 20])
def test_sorts_and_scans(ctx, n, limit):
    from sde_gb300 import _abi
    big = _job(ctx, 2048, 3 * n, 1)  # larger keys into the scratch
    assert _weights(ctx, *big, True)[0] == _abi.SDE_OK and _plan(ctx, *big)[0] == _abi.SDE_OK
    g, t = _job(ctx, 256, n, 2)
    want_w, want_p = _weights(ctx, g, t, True), _plan(ctx, g, t)
    assert want_w[0] == want_p[0] == _abi.SDE_OK
    assert _weights(ctx, *big, True)[0] == _abi.SDE_OK and _plan(ctx, *big)[0] == _abi.SDE_OK
    try:
        _abi.lib().sde_ctx_set_wait_limit(ctx.h, limit)
        got = [_weights(ctx, g, t, True), _weights(ctx, g, t, False)]
        plan = _plan(ctx, g, t)
    finally:
        _abi.lib().sde_ctx_set_wait_limit(ctx.h, -1)
    for rc, new, gwt in got:
        assert rc in (_abi.SDE_OK, _abi.SDE_ETIMEDOUT)
        if limit == 0:
            assert rc == (_abi.SDE_OK if n <= 2048 else _abi.SDE_ETIMEDOUT)
        if rc == _abi.SDE_OK:
            assert ctx.torch.equal(new, want_w[1]) and ctx.torch.equal(gwt, want_w[2])
        else:
            assert not new.any()
    assert plan[0] in (_abi.SDE_OK, _abi.SDE_ETIMEDOUT)
    if limit == 0:
        assert plan[0] == _abi.SDE_ETIMEDOUT
    ctx.sync()  # nothing is left over
    again_w, again_p = _weights(ctx, g, t, True), _plan(ctx, g, t)
    assert again_w[0] == again_p[0] == _abi.SDE_OK
    assert ctx.torch.equal(again_w[1], want_w[1]) and ctx.torch.equal(again_w[2], want_w[2])
    pk = want_p[1].abs().max()
    for p in [again_p] + ([plan] if plan[0] == _abi.SDE_OK else []):
        assert (p[1] - want_p[1]).abs().max() <= 1e-5 * pk  # (atomics add in any order)

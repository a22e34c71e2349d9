"""A pointing whose weight is infinite or NaN changes no mosaic pixel outside its own image."""
import ctypes as C

import numpy as np
import pytest

from conftest import small_obs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_weight_stays_in_its_image(gpu_ctx, bad):
    from sde_gb300._abi import check, lib
    from sde_gb300.mosaic import Mosaic
    pts = [dict(small_obs(imsize=64, cell=8.0, ntime=2, seed=3 + i), imsize=64, l0=0.0, m0=0.0, pb_fwhm_rad=0.01)
           for i in range(2)]
    m = Mosaic(gpu_ctx, pts, 8.0, mosaic=False)
    mnx, mny = 150, 130
    cx, cy, fw = np.array([50, 90], np.int32), np.array([50, 75], np.int32), np.full(2, 40.0, np.float32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    wt = np.array([bad, 1.0], np.float32)
    check(lib().sde_batch_set_mosaic(m.h, mnx, mny, p(cx), p(cy), p(fw), p(wt), 0.1), "sde_batch_set_mosaic")
    m.layout = dict(mnx=mnx, mny=mny)
    m.dirty(graph=False)
    out = m.read()
    m.close()
    inside = np.zeros((mny, mnx), bool)
    inside[50 - 32:50 + 32, 50 - 32:50 + 32] = True  # 64 x 64 about (cx - 1, cy - 1) = image pixel 31
    assert np.isfinite(out[~inside]).all()

"""The PI-original rebin of a detector that is wider than the source distance: a column with |s| > dso has
no ray, and its coordinates are NaN.  With border addressing it reads 0, as every sample outside the
detector does; with clamped addressing it stays NaN.  The other columns are the oracle's (tolerance of the
kernel's other tests: 1e-6, FP32 blends of FP64 geometry)."""
import ctypes as C

import numpy as np
import pytest

import oracle as orc
from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("addr", [capi.ADDR_BORDER, capi.ADDR_CLAMP])
def test_columns_past_the_source_distance(cuda, addr):
    import torch

    geo = ScanGeometry(ns=131, nt=9, ds=1.0, dt=1.0, npt=122, pitch=0.9, nx=16, ny=16, dx=1.0, dz=1.0).with_blocks(1)
    g = capi.Geom.from_buffer_copy(Plan(geo).info.ctg)
    g.dso = 50.5  # columns beyond 50 of 65 from the centre have no ray
    g.n_angle, g.n_angle_add = 70, 70 + 2 * g.add_projections
    fan = np.random.default_rng(2).standard_normal((g.n_angle_add, g.nt, g.ns)).astype(np.float32)
    d_fan = torch.from_numpy(fan).cuda()
    out = torch.full((g.n_angle, g.nt, g.ns), 7.0, device="cuda")
    capi.check(capi.lib().lct_rebin_pi_ori(C.byref(g), d_fan.data_ptr(), out.data_ptr(), capi.INTERP_EXACT,
                                           addr, None))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    outside = np.abs((np.arange(g.ns) - g.ws) * g.ds) > g.dso
    assert outside.any() and not outside.all()
    assert orc.rel_l2(got[:, :, ~outside], orc.rebin_pi_ori(g, fan, orc.EXACT, addr)[:, :, ~outside]) < 1e-6
    if addr == capi.ADDR_BORDER:
        assert (got[:, :, outside] == 0.0).all()
    else:
        assert np.isnan(got[:, :, outside]).all()

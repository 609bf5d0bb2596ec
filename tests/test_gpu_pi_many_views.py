"""The PI-original rebin and weight of more views than one launch of their grids holds (65,535 walks of 64
views), on a detector of 3 x 2: against the oracle with the kernels' tolerance (1e-6), the views at the
launches' seam and the last ones apart."""
import ctypes as C

import numpy as np
import pytest

import oracle as orc
from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


def test_more_views_than_a_launch(cuda):
    import torch

    geo = ScanGeometry(ns=3, nt=2, ds=8.0, dt=1.0, npt=122, pitch=0.9, nx=16, ny=16, dx=1.0,
                       dz=1.0).with_blocks(1)
    g = capi.Geom.from_buffer_copy(Plan(geo).info.ctg)
    g.n_angle = 65535 * 64 + 70
    g.n_angle_add = g.n_angle + 2 * g.add_projections
    fan = np.random.default_rng(6).standard_normal((g.n_angle_add, 2, 3)).astype(np.float32)
    d_fan = torch.from_numpy(fan).cuda()
    out = torch.full((g.n_angle, 2, 3), float("nan"), device="cuda")
    lib = capi.lib()
    capi.check(lib.lct_rebin_pi_ori(C.byref(g), d_fan.data_ptr(), out.data_ptr(), capi.INTERP_EXACT,
                                    capi.ADDR_BORDER, None))
    torch.cuda.synchronize()
    par = out.cpu().numpy()
    ref = orc.rebin_pi_ori(g, fan, orc.EXACT, capi.ADDR_BORDER)
    capi.check(lib.lct_weight_pi_ori(C.byref(g), out.data_ptr(), None))
    torch.cuda.synchronize()
    wgt, wref = out.cpu().numpy(), orc.weight_pi_ori(g, par)
    seam = 65535 * 64
    for views in (slice(None), slice(seam - 64, seam + 64), slice(g.n_angle - 8, None)):
        assert orc.rel_l2(par[views], ref[views]) < 1e-6
        assert orc.rel_l2(wgt[views], wref[views]) < 1e-6

"""The PI-original kernels where their tiles end: columns past a CTA's 128, rows, views past a walk of
64, slices past a chunk of 8 and an odd last pair, both addressings -- against the oracle.
Tolerances: the rebin's FP64 geometry and the weight 1e-6 (FP32 blends); the backprojector 1e-4 in
EXACT, the stage tests' bar (a view whose |t| falls within a rounding of pitch / 4 may be counted on
either side), and twice that in TEX8, whose 8-bit weights also move by a step where a coordinate's
rounding differs."""
import ctypes as C

import numpy as np
import pytest

import oracle as orc
from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def block(cuda):
    geo = ScanGeometry(ns=131, nt=9, ds=1.0, dt=1.0, npt=122, pitch=0.9, nx=37, ny=19, dx=1.5,
                       dz=0.8).with_blocks(1)
    p = Plan(geo)
    g, ig = p.info.ctg, p.info.ig
    rng = np.random.default_rng(3)
    v, t, s = np.ogrid[: g.n_angle_add, : g.nt, : g.ns]
    fan = (2.0 + np.sin(0.05 * v + 0.1 * s) * np.cos(0.3 * t) + 0.05 * rng.standard_normal(
        (g.n_angle_add, g.nt, g.ns))).astype(np.float32)
    b0 = p.blocks[0].block_proj_start + g.add_projections
    return g, ig, fan, np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])


@pytest.mark.parametrize("addr", [capi.ADDR_BORDER, capi.ADDR_CLAMP])
def test_rebin_and_weight(block, addr):
    import torch

    g, _, fan, _ = block
    lib = capi.lib()
    d_fan = torch.from_numpy(fan).cuda()
    out = torch.full((g.n_angle, g.nt, g.ns), float("nan"), device="cuda")
    capi.check(lib.lct_rebin_pi_ori(C.byref(g), d_fan.data_ptr(), out.data_ptr(), capi.INTERP_EXACT,
                                    addr, None))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert orc.rel_l2(got, orc.rebin_pi_ori(g, fan, orc.EXACT, addr)) < 1e-6
    capi.check(lib.lct_weight_pi_ori(C.byref(g), out.data_ptr(), None))
    torch.cuda.synchronize()
    assert orc.rel_l2(out.cpu().numpy(), orc.weight_pi_ori(g, got)) < 1e-6


@pytest.mark.parametrize("nz", [1, 7, 9, 32])
@pytest.mark.parametrize("interp,tol", [(capi.INTERP_EXACT, 1e-4), (capi.INTERP_TEX8, 2e-4)])
def test_backproject(block, nz, interp, tol):
    import torch

    g, ig, fan, betas = block
    ig = capi.Img.from_buffer_copy(ig)
    ig.nz = nz
    proj = np.ascontiguousarray(fan[: g.n_angle] - 2.0)
    d_proj, d_b = torch.from_numpy(proj).cuda(), torch.from_numpy(betas).cuda()
    for addr in (capi.ADDR_BORDER, capi.ADDR_CLAMP):
        img = torch.full((nz, ig.ny, ig.nx), float("nan"), device="cuda")
        capi.check(capi.lib().lct_backproject_pi_ori(C.byref(g), C.byref(ig), d_b.data_ptr(),
                                                     d_proj.data_ptr(), img.data_ptr(), interp, addr,
                                                     None))
        torch.cuda.synchronize()
        ref = orc.bp_pi_ori(g, ig, betas, proj, orc.TEXEMU if interp == capi.INTERP_TEX8 else orc.EXACT,
                            addr)
        assert orc.rel_l2(img.cpu().numpy(), ref) < tol

"""The exact PI-window walk over views that hold an infinite sample: a voxel that blends it is infinite of its sign, as
weights times texels have it (differences of texels would make it NaN); a NaN is left only where its weight
is exactly 0, in a few voxels in 100,000 (8-bit weights are 0 far more often).  Voxels that do not reach it are the same bits as without it."""
import ctypes as C

import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("addr", [capi.ADDR_BORDER, capi.ADDR_CLAMP])
def test_infinite_samples(cuda, addr):
    import torch

    nx = 144
    p = Plan(ScanGeometry(ns=96, nt=16, ds=1.0, dt=1.0, npt=120, pitch=1.2, nx=nx, ny=nx, dx=60.0 / nx,
                          dz=0.9).with_blocks(1))
    g, ig = p.info.ctg, p.info.ig
    b0 = p.blocks[0].block_proj_start + g.add_projections
    betas = torch.from_numpy(np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])).cuda()
    proj = torch.randn((g.n_angle, g.nt, g.ns), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))

    def run(x):
        out = torch.zeros((ig.nz, nx, nx), device="cuda")
        capi.check(capi.lib().lct_backproject_pi_ori(C.byref(g), C.byref(ig), betas.data_ptr(), x.data_ptr(),
                                                     out.data_ptr(), capi.INTERP_EXACT, addr, None))
        torch.cuda.synchronize()
        return out.cpu().numpy()

    clean = run(proj)
    mid = g.n_angle // 2
    for value in (float("inf"), -float("inf")):
        bad = proj.clone()
        bad[mid - 40:mid + 40:8, 4:12:3, 20:76:9] = value
        got = run(bad)
        finite = np.isfinite(got)
        assert np.array_equal(got[finite], clean[finite])
        assert (got == value).sum() > 100
        assert np.isnan(got).mean() < 1e-4 and (got == -value).sum() == 0

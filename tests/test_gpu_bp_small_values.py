"""TEX8 backprojection of views near the smallest floats: a scale of 2^-130 puts the samples below the smallest
normal number, where a sample is a multiple of 2^-149, and the volume then still is the unscaled one's to what
those multiples allow -- about 500 roundings of 2^-150 in a voxel's sum of some 4 x 2^-130 (120 samples of
random views): 1e-6 to 1e-5; tolerance 2e-5."""
import ctypes as C

import numpy as np
import pytest

import oracle as orc
from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [40, 144, 280])
def test_subnormal_views(cuda, nx):
    import torch

    p = Plan(ScanGeometry(ns=96, nt=16, ds=1.0, dt=1.0, npt=120, pitch=1.2, nx=nx, ny=nx, dx=60.0 / nx,
                          dz=0.9).with_blocks(1))
    g, ig = p.info.ctg, p.info.ig
    b0 = p.blocks[0].block_proj_start + g.add_projections
    betas = torch.from_numpy(np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])).cuda()
    # whole multiples of 2^-19, so that the scaled views are exact
    x = np.round(np.random.default_rng(3).standard_normal((g.n_angle, g.nt, g.ns)) * 2 ** 19)
    vols = []
    for scale in (2.0 ** -19, 2.0 ** -149):
        proj = torch.from_numpy((x * scale).astype(np.float32)).cuda()
        out = torch.zeros((ig.nz, nx, nx), device="cuda")
        capi.check(capi.lib().lct_backproject_par(C.byref(g), C.byref(ig), betas.data_ptr(), proj.data_ptr(),
                                                  out.data_ptr(), capi.INTERP_TEX8, capi.ADDR_BORDER, None))
        torch.cuda.synchronize()
        vols.append(out.cpu().numpy().astype(np.float64))
    assert orc.rel_l2(vols[1] * 2.0 ** 130, vols[0]) < 2e-5

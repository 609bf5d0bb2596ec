"""The exact backprojector's split over threads: a small image takes 1, 2 or 4 slices per thread where a
larger one takes 8, and every slice is rounded as in a thread of 8 (or of 4, where few slices are active
together), so a voxel's value depends on its own position alone.  The same tile-aligned corner of the
volume is backprojected as part of images on each side of the rule's lines and has to be the same bits.
Every image keeps the largest one's centre, so the corner's voxels coincide."""
import ctypes as C

import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pitch", [0.6, 1.5])
@pytest.mark.parametrize("nx", [48, 80, 144])  # 1, 2 and 4 slices per thread; 272: 8
def test_corner_of_images(cuda, nx, pitch):
    import torch

    # 0.5 mm voxels: the largest image's corner lies 96 mm from the axis, inside the fan
    geo = ScanGeometry(ns=272, nt=8, ds=1.0, dt=1.0, npt=120, pitch=pitch, nx=272, ny=272, dx=0.5,
                       dz=0.7).with_blocks(1)
    p = Plan(geo)
    g, ig = p.info.ctg, p.info.ig
    b0 = p.blocks[0].block_proj_start + g.add_projections
    rng = np.random.default_rng(5)
    proj = torch.from_numpy(rng.standard_normal((g.n_angle, g.nt, g.ns)).astype(np.float32)).cuda()
    betas = torch.from_numpy(np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])).cuda()

    def run(n):
        im = capi.Img.from_buffer_copy(ig)
        im.nx = im.ny = n
        out = torch.full((im.nz, n, n), float("nan"), device="cuda")
        capi.check(capi.lib().lct_backproject_par(C.byref(g), C.byref(im), betas.data_ptr(),
                                                  proj.data_ptr(), out.data_ptr(),
                                                  capi.INTERP_EXACT, capi.ADDR_BORDER, None))
        torch.cuda.synchronize()
        return out[:, :48, :48].cpu().numpy()

    assert np.array_equal(run(nx), run(272))

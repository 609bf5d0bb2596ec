"""The exact backprojector on partly filled view windows.  A thread's slices share each view, and
near the ends of their windows only some of them use it: the groups of slices that hold one run,
and the others' sums are left alone.  Slice counts around the chunk (8) and group (2) sizes, every
slices-per-thread shape, and a steep scan whose samples leave the detector rows -- against the
FP64 oracle of the same block.  Tolerance: TOL of the stage tests (1e-5), which the kernel's FP32
geometry reaches on this scan with full windows."""
import ctypes as C

import numpy as np
import pytest

import oracle as orc
from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


def _block(pitch, seed):
    geo = ScanGeometry(ns=96, nt=8, ds=1.0, dt=1.0, npt=120, pitch=pitch, nx=33, ny=18, dx=1.0,
                       dz=0.7).with_blocks(1)
    p = Plan(geo)
    g, ig = p.info.ctg, p.info.ig
    rng = np.random.default_rng(seed)
    v, t, s = np.ogrid[: g.n_angle, : g.nt, : g.ns]
    proj = (np.sin(0.05 * v + 0.1 * s) * np.cos(0.3 * t) + 0.05 * rng.standard_normal(
        (g.n_angle, g.nt, g.ns))).astype(np.float32)
    b0 = p.blocks[0].block_proj_start + g.add_projections
    return g, ig, proj, p.angles32[b0:b0 + g.n_angle]


@pytest.mark.parametrize("nz", [1, 2, 3, 7, 8, 9, 15, 32])
@pytest.mark.parametrize("pitch", [0.6, 1.5])
def test_partial_windows(cuda, nz, pitch):
    import torch

    g, ig, proj, betas = _block(pitch, 7)
    ig = capi.Img.from_buffer_copy(ig)
    ig.nz = nz
    d_proj, d_b = torch.from_numpy(proj).cuda(), torch.from_numpy(np.ascontiguousarray(betas)).cuda()
    for addr in (capi.ADDR_BORDER, capi.ADDR_CLAMP):
        img = torch.full((nz, ig.ny, ig.nx), float("nan"), device="cuda")
        capi.check(capi.lib().lct_backproject_par(C.byref(g), C.byref(ig), d_b.data_ptr(),
                                                  d_proj.data_ptr(), img.data_ptr(),
                                                  capi.INTERP_EXACT, addr, None))
        torch.cuda.synchronize()
        ref = orc.bp_par(g, ig, betas, proj, orc.EXACT, addr)
        assert orc.rel_l2(img.cpu().numpy(), ref) < 1e-5

"""Every thread shape of the backprojector on slice counts around the chunks (8, 4, 2 slices) and groups (2) of its
threads, on the partly filled windows of a scan with few active slices and of one with many: remainders of a
chunk, slices that are evaluated with their group and not added, both interpolations and addressings.  A voxel
is the same bits in an image of any size, so a 33 x 18 image, which takes one slice per thread (that shape is
what test_gpu_bp_windows holds to the FP64 oracle), is compared with the same voxels of larger images that
take 2, 4 and 8."""
import ctypes as C

import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

NX, NY = 33, 18
SIZES = (144, 272, 400, 560)


def _block(pitch, n, nz):
    """The block's geometry and an n x n (or the 33 x 18) image of it, every image with its first voxel in the
    same place."""
    p = Plan(ScanGeometry(ns=96, nt=8, ds=1.0, dt=1.0, npt=120, pitch=pitch, nx=NX, ny=NY, dx=0.25,
                          dz=0.7).with_blocks(1))
    ig = capi.Img.from_buffer_copy(p.info.ig)
    if n:
        ig.nx = ig.ny = n
    ig.nz = nz
    return p, p.info.ctg, ig


def _slices(pitch, n, nz):
    _, g, ig = _block(pitch, n, nz)
    out = C.c_int(-1)
    capi.check(capi.load().lct_backproject_par_slices(C.byref(g), C.byref(ig), 1, C.byref(out)))
    return out.value


@pytest.mark.parametrize("pitch,shapes", [(0.6, {1, 2, 4}), (1.5, {1, 2, 4, 8})])
def test_the_sizes_reach_every_shape(pitch, shapes):
    for nz in (7, 9, 15):
        assert _slices(pitch, 0, nz) == 1
    assert {_slices(pitch, n, nz) for n in SIZES for nz in (7, 9, 15)} | {1} == shapes
    if pitch == 1.5:  # 8 slices per thread with a remainder
        assert _slices(pitch, 560, 7) == _slices(pitch, 400, 9) == _slices(pitch, 400, 15) == 8


@pytest.mark.gpu
@pytest.mark.parametrize("nz", [1, 2, 3, 7, 8, 9, 15, 32])
@pytest.mark.parametrize("pitch", [0.6, 1.5])
@pytest.mark.parametrize("interp", [capi.INTERP_EXACT, capi.INTERP_TEX8])
def test_remainders(cuda, interp, pitch, nz):
    import torch

    p, g, small = _block(pitch, 0, nz)
    rng = np.random.default_rng(7)
    v, t, s = np.ogrid[: g.n_angle, : g.nt, : g.ns]
    proj = (np.sin(0.05 * v + 0.1 * s) * np.cos(0.3 * t) + 0.05 * rng.standard_normal(
        (g.n_angle, g.nt, g.ns))).astype(np.float32)
    b0 = p.blocks[0].block_proj_start + g.add_projections
    d_b = torch.from_numpy(np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])).cuda()
    d_proj = torch.from_numpy(proj).cuda()

    def run(ig, addr):
        out = torch.full((ig.nz, ig.ny, ig.nx), float("nan"), device="cuda")
        capi.check(capi.lib().lct_backproject_par(C.byref(g), C.byref(ig), d_b.data_ptr(), d_proj.data_ptr(),
                                                  out.data_ptr(), interp, addr, None))
        torch.cuda.synchronize()
        assert bool(torch.isfinite(out).all())
        return out[:, :NY, :NX].cpu().numpy()

    for addr in (capi.ADDR_BORDER, capi.ADDR_CLAMP):
        want = run(small, addr)
        for n in SIZES:
            assert np.array_equal(run(_block(pitch, n, nz)[2], addr), want), n

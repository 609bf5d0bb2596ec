"""A volume that reaches past the source's circle.  Voxels near it project to row coordinates beyond the range
of int (or to infinity), voxels past it have no ray in some views (NaN); with both addressings every sample
then has to stay inside the views.  A voxel's value depends on its own position alone, so the voxels of the
volume's central 16 x 16 tiles are the same bits as in a volume of those tiles, which ends inside the circle
(and which the other tests hold to the oracle)."""
import ctypes as C

import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("addr", [capi.ADDR_BORDER, capi.ADDR_CLAMP])
@pytest.mark.parametrize("interp", [capi.INTERP_EXACT, capi.INTERP_TEX8])
@pytest.mark.parametrize("window", ["par", "pi"])
def test_volume_past_the_source(cuda, window, interp, addr):
    import torch

    n, lo, m = 81, 16, 48  # columns, the central tiles' first and their number
    geo = ScanGeometry(ns=96, nt=8, ds=1.0, dt=1.0, npt=120, pitch=0.9, nx=n, ny=n, dx=1.5, dz=0.8,
                       dso=57.0).with_blocks(1)
    p = Plan(geo)
    g, ig = p.info.ctg, capi.Img.from_buffer_copy(p.info.ig)
    ig.nz = 9
    x, y = (np.arange(n) - ig.wx) * ig.dx, (np.arange(n) - ig.wy) * ig.dy
    r = np.hypot(x[None, :], y[:, None])
    assert np.isclose(r, g.dso).any() and r.max() > 1.3 * g.dso  # voxels on the circle and past it
    assert r[lo:lo + m, lo:lo + m].max() < 0.95 * g.dso
    v, t, s = np.ogrid[: g.n_angle, : g.nt, : g.ns]
    proj = torch.from_numpy((np.sin(0.05 * v + 0.1 * s) * np.cos(0.3 * t)).astype(np.float32)).cuda()
    b0 = p.blocks[0].block_proj_start + g.add_projections
    betas = torch.from_numpy(np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])).cuda()
    fn = capi.lib().lct_backproject_par if window == "par" else capi.lib().lct_backproject_pi_ori

    def run(im):
        out = torch.zeros((im.nz, im.ny, im.nx), device="cuda")
        capi.check(fn(C.byref(g), C.byref(im), betas.data_ptr(), proj.data_ptr(), out.data_ptr(), interp,
                      addr, None))
        torch.cuda.synchronize()
        return out.cpu().numpy()

    central = capi.Img.from_buffer_copy(ig)
    central.nx = central.ny = m
    central.wx, central.wy = ig.wx - lo, ig.wy - lo
    want = run(central)
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    assert np.array_equal(run(ig)[:, lo:lo + m, lo:lo + m], want)

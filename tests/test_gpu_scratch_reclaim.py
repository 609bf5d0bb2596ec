"""The scratch that the stage entry points keep between calls does not stand in the way of the process's
other allocations: one that is larger than what is free, but not than what is free and kept, gets the kept
memory; the next call takes its scratch again."""
import ctypes as C

import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


def test_another_allocation_gets_the_kept_scratch(cuda):
    import torch

    lib = capi.load()
    p = Plan(ScanGeometry(ns=736, nt=64, ds=0.6, dt=0.6, npt=1152, pitch=0.8, nx=32, ny=32, dx=1.0,
                          dz=1.0).with_blocks(1))
    g, ig = p.info.ctg, p.info.ig
    b0 = p.blocks[0].block_proj_start + g.add_projections
    betas = torch.from_numpy(np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])).cuda()
    proj = torch.randn((g.n_angle, g.nt, g.ns), device="cuda")
    img = torch.empty((ig.nz, ig.ny, ig.nx), device="cuda")

    def run():
        capi.check(lib.lct_backproject_par(C.byref(g), C.byref(ig), betas.data_ptr(), proj.data_ptr(),
                                           img.data_ptr(), capi.INTERP_EXACT, capi.ADDR_BORDER, None))
        torch.cuda.synchronize()
        return img.clone()

    capi.check(lib.lct_scratch_release())
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    want = run()
    free = torch.cuda.mem_get_info()[0]
    kept = before - free
    assert kept > 1 << 30  # the block's quads, 16 bytes a sample
    big = torch.empty(free + kept // 2, dtype=torch.uint8, device="cuda")
    assert big.numel() > free
    del big
    torch.cuda.empty_cache()
    assert torch.equal(run(), want)
    capi.check(lib.lct_scratch_release())

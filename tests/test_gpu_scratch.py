"""The stage entry points' scratch pool: memory kept between calls is bounded and goes back on
request, and calls on two streams at once do not share scratch (each volume equals its own
sequential run, bit for bit)."""
import ctypes as C

import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan

pytestmark = pytest.mark.gpu


def test_scratch_is_private_to_a_call_and_given_back(small_geo, cuda):
    import torch

    lib = capi.load()
    p = Plan(small_geo)
    g, ig = p.info.ctg, p.info.ig
    b0 = p.blocks[0].block_proj_start + g.add_projections
    betas = torch.from_numpy(np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])).cuda()
    gen = torch.Generator(device="cuda").manual_seed(5)
    projs = [torch.randn((g.n_angle, g.nt, g.ns), device="cuda", generator=gen) for _ in range(2)]

    def run(proj, stream):
        img = torch.empty((ig.nz, ig.ny, ig.nx), device="cuda")
        capi.check(lib.lct_backproject_par(C.byref(g), C.byref(ig), betas.data_ptr(), proj.data_ptr(),
                                           img.data_ptr(), capi.INTERP_EXACT, capi.ADDR_BORDER,
                                           stream.cuda_stream))
        return img

    torch.cuda.synchronize()
    one = torch.cuda.Stream()
    refs = []
    for x in projs:
        refs.append(run(x, one))
        torch.cuda.synchronize()
    two = torch.cuda.Stream()
    for _ in range(5):
        outs = [run(x, s) for x, s in zip(projs, (one, two))]
        torch.cuda.synchronize()
        assert all(torch.equal(o, r) for o, r in zip(outs, refs))
    before = torch.cuda.mem_get_info()[0]
    capi.check(lib.lct_scratch_release())
    after = torch.cuda.mem_get_info()[0]
    assert after > before  # this block's quads were kept
    capi.check(lib.lct_scratch_release())
    out = run(projs[0], one)  # and the pool serves the next call
    torch.cuda.synchronize()
    assert torch.equal(out, refs[0])

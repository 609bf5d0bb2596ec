"""Options of the backprojector on small images, where the default takes one slice per thread: a register budget
or the TMA-staged sampler that is asked for is what runs (a block-mode recon's autotuner, which has nothing
to tune, tells the shape), with the default's values."""
import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan, Reconstruction
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts,shape", [({}, (1, 4)), (dict(bp_minb=2), (8, 2)), (dict(bp_minb=4), (1, 4)),
                                        (dict(bp_sampler=capi.BP_SAMPLER_QUADS_TMA), (8, 4)),
                                        (dict(bp_nz=4), (4, 4))])
def test_what_is_asked_for_runs(cuda, opts, shape):
    import torch

    p = Plan(ScanGeometry(ns=96, nt=16, ds=1.0, dt=1.0, npt=120, pitch=1.0, nx=32, ny=29, dx=1.25,
                          dz=1.0).with_blocks(1))
    kw = dict(interp=capi.INTERP_EXACT, filter_mode=capi.FILTER_BF16X6, addr=capi.ADDR_BORDER)
    block = Reconstruction(p, mode=capi.MODE_BLOCK, **kw, **opts)
    assert block.autotune() == shape
    if opts.get("bp_nz"):
        return  # a requested number of slices has a base of its own
    for mode in (capi.MODE_BLOCK, capi.MODE_SCAN):
        rec, ref = Reconstruction(p, mode=mode, **kw, **opts), Reconstruction(p, mode=mode, **kw)
        g = p.info.ctg
        gen = torch.Generator(device="cuda").manual_seed(4)
        fan = torch.randn((ref.fan_first + ref.fan_count, g.nt, g.ns), device="cuda", generator=gen)
        assert np.array_equal(rec.run(fan).cpu().numpy(), ref.run(fan).cpu().numpy())

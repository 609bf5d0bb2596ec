"""The backprojection autotuner on small images, where the default takes fewer slices per thread than can be
requested: asking for tuning is not slower than not asking (a fifth at most, the best of several runs each; with
4, 8 and 16 slices alone it took twice the default's time), the values are the default's, and in a batch a
scan whose default is of another kind than the tuned scan's keeps its own."""
import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Batch, Plan, Reconstruction
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


def _plan(nx, blocks, dz=1.0):
    return Plan(ScanGeometry(ns=512, nt=16, ds=0.19, dt=1.0, npt=1000, pitch=1.0, nx=nx, ny=nx, dx=40.0 / nx,
                             dz=dz).with_blocks(blocks))


def _fan(plan, seed):
    import torch

    r = Reconstruction(plan)
    g = plan.info.ctg
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((r.fan_first + r.fan_count, g.nt, g.ns), device="cuda", generator=gen)


def _best(run, times):
    run()
    out = []
    for _ in range(6):
        run()
        out.append(times()["backproject"])
    return min(out)


@pytest.mark.parametrize("interp", [capi.INTERP_EXACT, capi.INTERP_TEX8])
@pytest.mark.parametrize("nx", [32, 64])
def test_tuning_a_small_image(cuda, nx, interp):
    p = _plan(nx, 1)
    kw = dict(mode=capi.MODE_SCAN, interp=interp, filter_mode=capi.FILTER_BF16X6)
    fan = _fan(p, nx)
    plain, tuned = Reconstruction(p, **kw), Reconstruction(p, bp_nz=-1, **kw)
    assert np.array_equal(tuned.run(fan).cpu().numpy(), plain.run(fan).cpu().numpy())
    a, b = _best(lambda: plain.run(fan), plain.last_times), _best(lambda: tuned.run(fan), tuned.last_times)
    assert b < 1.2 * a, (a, b)


def test_tuning_a_batch(cuda):
    plans = [_plan(32, 1), _plan(48, 1), _plan(32, 1, dz=1.5)]  # the last: few active slices
    kw = dict(interp=capi.INTERP_TEX8, filter_mode=capi.FILTER_BF16X6)
    fans = [_fan(p, 3 + i) for i, p in enumerate(plans)]
    plain, tuned = Batch(plans, **kw), Batch(plans, bp_nz=-1, **kw)
    for x, y in zip(tuned.run(fans), plain.run(fans)):
        assert np.array_equal(x.cpu().numpy(), y.cpu().numpy())
    a, b = _best(lambda: plain.run(fans), plain.last_times), _best(lambda: tuned.run(fans), tuned.last_times)
    assert b < 1.2 * a, (a, b)

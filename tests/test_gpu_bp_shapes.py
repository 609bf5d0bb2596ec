"""Backprojection thread shapes: the default by what runs together (one launch's slabs, a batch's scans).

A whole run, a streamed one (slab by slab), a bounded one (slab by slab from rings) and a batch (one work
list per shape) may each take another number of slices per thread -- with a base shared by threads of
fewer slices in EXACT -- and every one has to give the bits of 8 slices per thread.  And the default is not
slower than a requested shape by more than a fifth where many slabs or scans of a small image run together
(the best of several runs each; with the shape picked by one slab it was 1.5 times and more)."""
import ctypes as C

import numpy as np
import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Batch, Plan, Reconstruction
from listctrecons_b200.scan import ScanGeometry

pytestmark = pytest.mark.gpu


def _plan(nx, blocks, dz=1.0, ns=96, npt=120):
    return Plan(ScanGeometry(ns=ns, nt=16, ds=96.0 / ns, dt=1.0, npt=npt, pitch=1.0, nx=nx, ny=nx - 3,
                             dx=40.0 / nx, dz=dz).with_blocks(blocks))


def _fan(rec, seed):
    import torch

    g = rec.plan.info.ctg
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((rec.fan_first + rec.fan_count, g.nt, g.ns), device="cuda", generator=gen)


def _slices(plan, slabs):
    out = C.c_int(-1)
    capi.check(capi.load().lct_backproject_par_slices(C.byref(plan.info.ctg), C.byref(plan.info.ig), slabs,
                                                      C.byref(out)))
    return out.value


# columns, slabs, slices per thread of the whole launch and of one slab's
@pytest.mark.parametrize("nx,blocks,whole,slab", [(32, 3, 1, 1), (64, 2, 2, 2), (80, 2, 4, 2), (80, 3, 8, 2), (128, 3, 4, 4),
                                                  (128, 4, 8, 4), (192, 3, 8, 8)])
@pytest.mark.parametrize("interp", [capi.INTERP_EXACT, capi.INTERP_TEX8])
def test_every_run_gives_the_bits_of_eight_slices(cuda, nx, blocks, whole, slab, interp):
    import torch

    p = _plan(nx, blocks)
    assert (_slices(p, blocks), _slices(p, 1)) == (whole, slab)
    kw = dict(mode=capi.MODE_SCAN, interp=interp, filter_mode=capi.FILTER_BF16X6, addr=capi.ADDR_BORDER)
    rec = Reconstruction(p, **kw)
    fan = _fan(rec, 3)
    want = Reconstruction(p, bp_nz=8, **kw).run(fan).cpu().numpy()
    assert np.isfinite(want).all()
    assert np.array_equal(rec.run(fan).cpu().numpy(), want)
    h_fan = fan.cpu().pin_memory()
    h_img = torch.full(rec.image_shape, float("nan"), dtype=torch.float32).pin_memory()
    rec.run(h_fan, h_img)  # streamed, the first slab in parts
    assert np.array_equal(h_img.numpy(), want)
    bounded = Reconstruction(p, bounded=True, piece_views=24, **kw)
    h_img.fill_(float("nan"))
    bounded.run(h_fan, h_img)
    assert np.array_equal(h_img.numpy(), want)


# scans (columns, slabs, slice spacing); 1.5 mm: few active slices, a base of 4
@pytest.mark.parametrize("scans", [
    [(32, 1, 1.0), (24, 1, 1.5)],                   # 1 slice per thread, bases of 8 and 4
    [(64, 1, 1.0), (48, 1, 1.0), (32, 1, 1.5)],     # 2
    [(96, 1, 1.0), (80, 1, 1.0), (48, 1, 1.5)],     # 4, based and not
    [(144, 2, 1.0), (192, 1, 1.0), (96, 1, 1.5)],   # 8 and 4
])
@pytest.mark.parametrize("interp", [capi.INTERP_EXACT, capi.INTERP_TEX8])
def test_a_batch_gives_the_bits_of_single_runs(cuda, scans, interp):
    plans = [_plan(*s) for s in scans]
    kw = dict(interp=interp, filter_mode=capi.FILTER_BF16X6)
    b = Batch(plans, **kw)
    recs = [Reconstruction(p, **kw) for p in plans]
    fans = [_fan(r, 5 + i) for i, r in enumerate(recs)]
    for img, r, fan in zip(b.run(fans), recs, fans):
        assert np.array_equal(img.cpu().numpy(), r.run(fan).cpu().numpy())


def _best(run, times):
    run()
    out = []
    for _ in range(6):
        run()
        out.append(times()["backproject"])
    return min(out)


def test_default_shape_of_many_slabs_is_not_slow(cuda):
    p = _plan(48, 16, ns=512, npt=1000)
    kw = dict(mode=capi.MODE_SCAN, interp=capi.INTERP_EXACT, filter_mode=capi.FILTER_BF16X6)
    rec = Reconstruction(p, **kw)
    fan = _fan(rec, 1)
    ms = {}
    for nz in (0, 4, 8):
        r = Reconstruction(p, bp_nz=nz, **kw)
        ms[nz] = _best(lambda: r.run(fan), r.last_times)
    assert ms[0] < 1.2 * min(ms[4], ms[8]), ms


def test_default_shape_of_a_batch_is_not_slow(cuda):
    plans = [_plan(48, 4, ns=512, npt=1000) for _ in range(4)]
    ms, fans = {}, None
    for nz in (0, 4, 8):
        b = Batch(plans, interp=capi.INTERP_EXACT, filter_mode=capi.FILTER_BF16X6, bp_nz=nz)
        if fans is None:
            rec = Reconstruction(plans[0])
            fans = [_fan(rec, 7)] * 4
        ms[nz] = _best(lambda: b.run(fans), b.last_times)
    assert ms[0] < 1.2 * min(ms[4], ms[8]), ms

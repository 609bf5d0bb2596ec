"""The default number of slices per backprojection thread, by what one launch holds: a small image of one
slab takes few (the views' latency in series is what counts), the same image of many slabs takes all of a
base's slices, since the chip is full and a thread's view terms are shared best."""
import ctypes as C

import pytest

from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry


def _slices(nx, slabs, nz=32, dz=1.0):
    p = Plan(ScanGeometry(ns=96, nt=16, ds=1.0, dt=1.0, npt=120, pitch=1.0, nx=nx, ny=nx, dx=40.0 / nx,
                          dz=dz).with_blocks(1))
    ig = capi.Img.from_buffer_copy(p.info.ig)
    ig.nz = nz
    out = C.c_int(-1)
    capi.check(capi.load().lct_backproject_par_slices(C.byref(p.info.ctg), C.byref(ig), slabs, C.byref(out)))
    return out.value


@pytest.mark.parametrize("nx,slabs,want", [
    (32, 1, 1), (48, 1, 1), (64, 1, 2), (96, 1, 2), (128, 1, 4), (160, 1, 8), (192, 1, 8), (512, 1, 8),
    (32, 16, 4), (48, 16, 8), (96, 4, 8), (96, 16, 8), (128, 2, 4), (128, 4, 8), (160, 2, 4), (256, 8, 8)])
def test_shape_by_the_tiles_of_the_launch(nx, slabs, want):
    assert _slices(nx, slabs) == want


@pytest.mark.parametrize("nx,slabs,want", [(32, 1, 1), (96, 1, 2), (128, 1, 2), (192, 1, 4), (48, 16, 4),
                                           (96, 16, 4)])
def test_few_active_slices(nx, slabs, want):
    assert _slices(nx, slabs, dz=1.5) == want  # 16 mm of feed: 5.3 slices of 1.5 mm active


@pytest.mark.parametrize("nx,nz,want", [(512, 3, 4), (512, 5, 8), (512, 8, 8), (256, 5, 4), (33, 5, 1)])
def test_few_slices(nx, nz, want):
    assert _slices(nx, 1, nz=nz) == want  # 512^2 x 5: 1.61 ms in threads of 8, 1.84 ms in threads of 2


@pytest.mark.parametrize("nx", [32, 128, 512])
def test_never_more_threads_slices_than_a_few_slices_need(nx):
    assert _slices(nx, 1, nz=1) == 1
    assert _slices(nx, 1, nz=2) <= 2


def test_arguments():
    lib, out = capi.load(), C.c_int(-1)
    p = Plan(ScanGeometry(ns=96, nt=16, ds=1.0, dt=1.0, npt=120, pitch=1.0, nx=32, ny=32, dx=1.0,
                          dz=1.0).with_blocks(1))
    g, ig = p.info.ctg, p.info.ig
    assert lib.lct_backproject_par_slices(C.byref(g), C.byref(ig), 0, C.byref(out)) == capi.LCT_ERR_ARG
    assert lib.lct_backproject_par_slices(C.byref(g), C.byref(ig), 1, None) == capi.LCT_ERR_ARG
    assert lib.lct_backproject_par_slices(None, C.byref(ig), 1, C.byref(out)) == capi.LCT_ERR_ARG

"""The stage entry points after cudaDeviceReset (in a process of its own: it ends torch's context too): what
the library keeps per device -- the scratch pool, kernel attributes, the status word's address -- went with
the old context, and the calls give the same results in the new one, on new buffers."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
import ctypes as C
import sys
import numpy as np
from listctrecons_b200 import capi
from listctrecons_b200.recon import Plan
from listctrecons_b200.scan import ScanGeometry

rt = C.CDLL(sys.argv[1])
lib = capi.load()
p = Plan(ScanGeometry(ns=333, nt=8, ds=0.5, dt=0.5, npt=120, pitch=1.0, nx=32, ny=32, dx=1.0,
                      dz=0.5).with_blocks(1))
g, ig = p.info.ctg, p.info.ig
b0 = p.blocks[0].block_proj_start + g.add_projections
betas = np.ascontiguousarray(p.angles32[b0:b0 + g.n_angle])
views = np.random.default_rng(1).standard_normal((g.n_angle, g.nt, g.ns)).astype(np.float32)
taps = np.zeros(2 * g.ns, np.float32)
capi.check(lib.lct_filter_taps(capi.FILTER_RAMLAK, capi.WINDOW_NONE, g.ns, np.float32(g.ds), taps.ctypes.data))


def ok(e):
    assert e == 0, e


def put(a):
    d = C.c_void_p()
    ok(rt.cudaMalloc(C.byref(d), C.c_size_t(a.nbytes)))
    ok(rt.cudaMemcpy(d, C.c_void_p(a.ctypes.data), C.c_size_t(a.nbytes), 1))
    return d


def chain():
    d_h, d_b, d_v = put(taps), put(betas), put(views)
    img = np.full((ig.nz, ig.ny, ig.nx), np.nan, np.float32)
    d_i, out = put(img), []
    for mode in (capi.FILTER_FP32, capi.FILTER_BF16X6):
        capi.check(lib.lct_filter_rows(g.ns, d_h, d_v, g.n_angle * g.nt, mode, None))
        capi.check(lib.lct_backproject_par(C.byref(g), C.byref(ig), d_b, d_v, d_i, capi.INTERP_EXACT,
                                           capi.ADDR_BORDER, None))
        ok(rt.cudaMemcpy(C.c_void_p(img.ctypes.data), d_i, C.c_size_t(img.nbytes), 2))
        out.append(img.copy())
    code = C.c_int(-1)
    capi.check(lib.lct_device_status(C.byref(code)))
    assert code.value == 0
    capi.check(lib.lct_scratch_release())
    return np.stack(out)


first = chain()
assert np.isfinite(first).all()
ok(rt.cudaDeviceReset())
capi.check(lib.lct_scratch_release())  # nothing kept in the new context
second = chain()
assert np.array_equal(first, second)
"""


def test_calls_after_a_device_reset(cuda):
    lib = next(Path("/usr/local/cuda/lib64").glob("libcudart.so.12"))
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(lib)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr

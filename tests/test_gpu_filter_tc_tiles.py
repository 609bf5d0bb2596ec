"""The tensor-core filter where its tiles end: row blocks of 128, column tiles of 256 whose last one is
narrower, K slices of 32, planes padded to 8 samples, unaligned row widths, more tiles than SMs --
against the FP64 oracle, with the tolerances of the mode's other tests (BF16x6 1e-5, BF16x3 2e-4)."""
import ctypes as C

import numpy as np
import pytest

import oracle as orc
from listctrecons_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,tol", [(capi.FILTER_BF16X3, 2e-4), (capi.FILTER_BF16X6, 1e-5)])
@pytest.mark.parametrize("ns,nrows", [(9, 5), (31, 128), (33, 129), (255, 127), (256, 300), (257, 129),
                                      (511, 64), (735, 1000), (736, 19000), (1025, 130)])
def test_tiles(cuda, ns, nrows, mode, tol):
    import torch

    rng = np.random.default_rng(ns)
    x = np.linspace(0, 6, ns)
    rows = (2 + np.sin(x[None, :] * rng.uniform(0.5, 2, (nrows, 1))) +
            0.05 * rng.standard_normal((nrows, ns))).astype(np.float32)
    h = orc.shepp_logan_taps(ns, 0.6)
    d_rows, d_h = torch.from_numpy(rows).cuda(), torch.from_numpy(np.ascontiguousarray(h)).cuda()
    capi.check(capi.load().lct_filter_rows(ns, d_h.data_ptr(), d_rows.data_ptr(), nrows, mode, None))
    torch.cuda.synchronize()
    got = d_rows.cpu().numpy()
    keep = np.unique(np.concatenate([np.arange(min(nrows, 200)), np.arange(max(0, nrows - 200), nrows)]))
    assert orc.rel_l2(got[keep], orc.filter_rows_fp64(h, rows[keep])) < tol
    code = C.c_int(-1)
    assert capi.load().lct_device_status(C.byref(code)) == capi.LCT_OK and code.value == 0

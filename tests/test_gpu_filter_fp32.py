"""The FP32 ramp filter bit for bit in the reference's summation order, where its tiles end: eight
outputs and eight rows per thread, taps unrolled by eight, warps that hold the ends of two row
groups, more columns than a CTA has threads, unaligned row widths."""
import numpy as np
import pytest

import oracle as orc
from listctrecons_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nrows", [(1, 3), (5, 9), (7, 8), (8, 1), (9, 17), (15, 300), (96, 4000),
                                      (333, 37), (672, 500), (735, 129), (1000, 16), (2047, 5),
                                      (2056, 9), (3072, 3)])
def test_filter_fp32_bit_exact_at_tile_edges(cuda, ns, nrows):
    import torch

    rng = np.random.default_rng(ns)
    rows = rng.standard_normal((nrows, ns)).astype(np.float32)
    h = rng.standard_normal(2 * ns).astype(np.float32)
    d_rows, d_h = torch.from_numpy(rows).cuda(), torch.from_numpy(h).cuda()
    capi.check(capi.lib().lct_filter_rows(ns, d_h.data_ptr(), d_rows.data_ptr(), nrows,
                                          capi.FILTER_FP32, None))
    torch.cuda.synchronize()
    assert np.array_equal(d_rows.cpu().numpy(), orc.filter_rows(h, rows, mode=1).astype(np.float32))

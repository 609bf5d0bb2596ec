"""The network's kernels where their tiles end: convolution tiles of 8 rows x 128 pixels in blocks of 8,
gradient tiles of 6 rows x 64 pixels in groups of 3 and 16, images narrower than a block -- forward and
gradients against the FP64 oracle with the same bf16 storage points.  Tolerances: those of the network's
other tests (5e-3 forward, 2e-2 per layer of the gradients: what a changed summation order can do to
seven bf16 layers; an indexing error is of order one).  And a NaN pixel reaches the residual only within
the network's 17 x 17 window."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


def _params(seed):
    from listctrecons_b200.learn import N_PARAMS, layer_slices

    rng = np.random.default_rng(seed)
    p = np.zeros(N_PARAMS, dtype=np.float32)
    for ws, bs, shape in layer_slices():
        p[ws] = rng.normal(0.0, np.sqrt(2.0 / (9 * shape[1])), size=ws.stop - ws.start)
        p[bs] = rng.normal(0.0, 0.05, size=bs.stop - bs.start)
    return p


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 7), (1, 8, 8), (3, 9, 15), (1, 6, 63), (1, 7, 65),
                                   (1, 5, 127), (1, 17, 129), (2, 4, 130), (1, 3, 257)])
def test_forward_and_gradients_at_tile_edges(cuda, shape):
    import torch

    from listctrecons_b200.learn import CNN, layer_slices

    B, H, W = shape
    rng = np.random.default_rng(W)
    p = _params(4)
    x = rng.normal(0.5, 0.3, size=(B, 5, H, W)).astype(np.float32)
    t = rng.normal(0.4, 0.3, size=(B, H, W)).astype(np.float32)
    cnn = CNN(B, H, W, train=True)
    cnn.set_params(p)
    cnn.set_scales(0.8, 1.25)
    k_in = float(np.float32(0.8) * np.float32(1.25))
    xd, td = torch.as_tensor(x, device="cuda"), torch.as_tensor(t, device="cuda")
    r = cnn.forward(xd).cpu().numpy()
    assert orc.rel_l2(r, orc.cnn_forward(p.astype(np.float64), x, k_in, bf16=True)) < 5e-3
    cnn.backward(xd, td)
    g = cnn.grads()
    _, ref = orc.cnn_loss_grad(p.astype(np.float64), x, t, k_in, 1.25, bf16=True)
    for l, (ws, bs, _) in enumerate(layer_slices()):
        assert orc.rel_l2(g[ws], ref[ws]) < 2e-2, l
        assert orc.rel_l2(g[bs], ref[bs]) < 2e-2, l


def test_a_nan_stays_in_its_window(cuda):
    import torch

    from listctrecons_b200.learn import CNN

    B, H, W = 1, 40, 150
    rng = np.random.default_rng(8)
    x = rng.normal(0.5, 0.3, size=(B, 5, H, W)).astype(np.float32)
    cnn = CNN(B, H, W, train=True)
    cnn.set_params(_params(5))
    clean = cnn.forward(torch.as_tensor(x, device="cuda")).cpu().numpy()
    y, c = 19, 126
    x[0, 2, y, c] = np.nan
    got = cnn.forward(torch.as_tensor(x, device="cuda")).cpu().numpy()
    far = np.ones((H, W), dtype=bool)
    far[y - 8:y + 9, c - 8:c + 9] = False
    assert np.array_equal(got[0][far], clean[0][far])

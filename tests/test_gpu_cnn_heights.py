"""The convolution's tile heights: 8 output rows, and 4 or 2 where a launch has few tiles (the fewest rows whose
tiles are at most one for each SM).  A slice's residual is the same bits in a batch of any size, and forward
and gradients are the FP64 oracle's at the edges of every height (rows one past a tile, one short of it, widths
of one and two tiles; tolerances of the network's other tile tests: 5e-3 forward, 2e-2 per layer)."""
import numpy as np
import pytest

import oracle as orc
from tests.test_gpu_cnn_tiles import _params

pytestmark = pytest.mark.gpu


def _height(B, H, W, sms):
    tiles_x = (W + 127) // 128
    return next((r for r in (2, 4) if B * tiles_x * -(-H // r) <= sms), 8)


@pytest.mark.parametrize("H,W,batches", [(17, 9, {8: 40, 4: 20, 2: 2}), (15, 33, {8: 48, 4: 24, 2: 3}),
                                         (9, 129, {8: 26, 4: 20, 2: 4}), (5, 8, {8: 80, 4: 60, 2: 1})])
def test_every_height(cuda, H, W, batches):
    import torch

    from listctrecons_b200.learn import CNN, layer_slices

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = max(batches.values())
    rng = np.random.default_rng(H + W)
    p = _params(4)
    x = rng.normal(0.5, 0.3, size=(B, 5, H, W)).astype(np.float32)
    t = rng.normal(0.4, 0.3, size=(B, H, W)).astype(np.float32)
    cnn = CNN(B, H, W, train=True)
    cnn.set_params(p)
    cnn.set_scales(0.8, 1.25)
    k_in = float(np.float32(0.8) * np.float32(1.25))
    xd, td = torch.as_tensor(x, device="cuda"), torch.as_tensor(t, device="cuda")
    full = cnn.forward(xd).cpu().numpy()
    assert orc.rel_l2(full, orc.cnn_forward(p.astype(np.float64), x, k_in, bf16=True)) < 5e-3
    for height, n in batches.items():
        assert _height(n, H, W, sms) == height
        assert np.array_equal(cnn.forward(xd[:n].contiguous()).cpu().numpy(), full[:n])
        cnn.backward(xd[:n].contiguous(), td[:n].contiguous())
        g = cnn.grads()
        _, ref = orc.cnn_loss_grad(p.astype(np.float64), x[:n], t[:n], k_in, 1.25, bf16=True)
        for l, (ws, bs, _) in enumerate(layer_slices()):
            assert orc.rel_l2(g[ws], ref[ws]) < 2e-2, (height, l)
            assert orc.rel_l2(g[bs], ref[bs]) < 2e-2, (height, l)


def test_inference_of_few_and_many_slices(cuda):
    import torch

    from listctrecons_b200.learn import CNN

    H, W, nz = 21, 140, 40
    vol = torch.randn((nz, H, W), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    outs = []
    for cap in (1, 8, 32):  # passes of 1, 8 and 32 slices: tiles of 2, 4 and 8 rows
        cnn = CNN(cap, H, W, train=False)
        cnn.set_params(_params(6))
        cnn.set_scales(0.5, 2.0)
        outs.append(cnn.infer_volume(vol, bound=1e9)[0].cpu().numpy())
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


def test_one_slice_is_not_slow(cuda):
    """One 128 x 128 slice has a quarter of the work of four and leaves the chip emptier: its forward pass takes less
    than 0.9 of their time (0.98 with tiles of eight rows alone).  Graphs of ten passes, so that the host's
    launches do not count; the best of ten replays each."""
    import torch

    from listctrecons_b200.learn import CNN

    cnn = CNN(4, 128, 128, train=True)
    x = torch.randn((4, 5, 128, 128), device="cuda")
    out = torch.empty((4, 128, 128), device="cuda")

    def best(n):
        cnn.forward(x[:n], out[:n])
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(10):
                cnn.forward(x[:n], out[:n])
        ts = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return min(ts)

    one, four = best(1), best(4)
    print(one, four)
    assert one < 0.9 * four, (one, four)

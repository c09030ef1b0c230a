"""Convolutions over pixel boxes that reach past the images, against the plain
gathers.  Forward: weights of 0 and 1 and small whole inputs, so every sum is a
whole number below 2^24 and both paths must agree on every pixel.  Gradients:
layer by layer, every layer within the bound that test_gpu_unet_ragged.py sets
for all of them together."""
import numpy as np
import pytest

import airtoolsii_b200 as airt

from test_gpu_unet import _set_gemm_path

pytestmark = pytest.mark.gpu

SHAPES = [(6, 10, 16, 2, 1), (2, 2, 16, 2, 3), (12, 24, 32, 3, 5), (20, 48, 16, 3, 2), (10, 96, 32, 2, 3),
          (130, 14, 16, 2, 1), (40, 40, 48, 3, 2), (66, 130, 16, 2, 1), (66, 66, 32, 2, 3)]


def on_both_paths(f):
    out = []
    for path in (0, 1):
        _set_gemm_path(path)
        try:
            out.append(f())
        finally:
            _set_gemm_path(0)
    return out


@pytest.mark.parametrize("H,W,base,levels,B", SHAPES)
def test_forward_pixel_by_pixel(H, W, base, levels, B):
    import torch
    rng = np.random.default_rng(H * W + B)
    net = airt.UNet(H, W, base, levels, max_batch=B, seed=1)
    prm = []
    for cin, cout in net.layer_shapes():
        w = np.zeros((cout, 9 * cin), np.float32)
        for row in w:                                  # a few ones per channel, the first one a border tap
            row[rng.choice([0, 2, 6, 8]) * cin + rng.integers(cin)] = 1.0
            row[rng.integers(0, 9 * cin, 2)] = 1.0
        prm += [w.ravel(), np.zeros(cout, np.float32)]
    prm += [np.ones(base, np.float32), np.zeros(1, np.float32)]
    net.set_params(np.concatenate(prm))
    u = torch.as_tensor(rng.integers(0, 4, (B, H, W)).astype(np.float32)).cuda()

    def run():
        o = torch.zeros(B, H, W, device="cuda")
        net.forward(u.data_ptr(), o.data_ptr(), B)
        torch.cuda.synchronize()
        return o.cpu().numpy()
    a, b = on_both_paths(run)
    assert 0 < np.abs(b).max() < 2 ** 24
    assert np.array_equal(a, b)


@pytest.mark.parametrize("H,W,base,levels,B", SHAPES)
def test_gradients_layer_by_layer(H, W, base, levels, B):
    import torch
    gen = torch.Generator().manual_seed(H * W + 1)
    u = torch.randn(B, H, W, generator=gen).cuda()
    t = torch.randn(B, H, W, generator=gen).cuda()
    net = airt.UNet(H, W, base, levels, max_batch=B, seed=3)

    def run():
        net.gradients(u.data_ptr(), t.data_ptr(), B)
        return net.get_grads().astype(np.float64)
    a, b = on_both_paths(run)
    at = 0
    for cin, cout in net.layer_shapes():
        for n in (9 * cin * cout, cout):
            x, y = a[at:at + n], b[at:at + n]
            assert np.linalg.norm(x - y) <= 2e-2 * np.linalg.norm(y), (cin, cout, n)
            at += n
    assert np.linalg.norm(a[at:] - b[at:]) <= 2e-2 * np.linalg.norm(b[at:])

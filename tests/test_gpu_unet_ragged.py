"""Image sizes that no 128-pixel box tiles exactly: boxes reaching past the
rows, the columns and the last image, against the plain gathers."""
import numpy as np
import pytest

import airtoolsii_b200 as airt

from test_gpu_unet import _set_gemm_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,base,levels,B", [(6, 10, 16, 2, 1), (2, 2, 16, 2, 3), (12, 24, 32, 3, 5),
                                             (20, 48, 16, 3, 2), (10, 96, 32, 2, 3), (4, 192, 64, 2, 1),
                                             (130, 14, 16, 2, 1), (40, 40, 48, 3, 2), (66, 130, 16, 2, 1)])
def test_ragged_images(H, W, base, levels, B):
    import torch
    gen = torch.Generator().manual_seed(H * W)
    u = torch.randn(B, H, W, generator=gen).cuda()
    t = torch.randn(B, H, W, generator=gen).cuda()
    net = airt.UNet(H, W, base, levels, max_batch=B, seed=3)
    g, out = [], []
    for path in (0, 1):
        _set_gemm_path(path)
        try:
            o = torch.zeros(B, H, W, device="cuda")
            net.forward(u.data_ptr(), o.data_ptr(), B)
            torch.cuda.synchronize()
            out.append(o.cpu().numpy().astype(np.float64))
            net.gradients(u.data_ptr(), t.data_ptr(), B)
            g.append(net.get_grads().astype(np.float64))
        finally:
            _set_gemm_path(0)
    # BF16 roundings can flip on the order of the FP32 sums
    assert np.linalg.norm(out[0] - out[1]) <= 1e-2 * np.linalg.norm(out[1])
    assert np.linalg.norm(g[0] - g[1]) <= 2e-2 * np.linalg.norm(g[1])

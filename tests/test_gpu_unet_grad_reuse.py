"""The activations' gradient buffers are not zeroed between calls: the first
writer of each stores every element.  A second call, with another batch size,
has to give what a network that never ran before gives."""
import numpy as np
import pytest

import airtoolsii_b200 as airt

pytestmark = pytest.mark.gpu


# small images (plain tiles), 128 pixels wide (row strips), 16 base channels
# (32-byte rows) and 4 levels
@pytest.mark.parametrize("H,W,base,levels", [(16, 16, 16, 2), (32, 128, 32, 3), (24, 128, 16, 2),
                                             (16, 128, 64, 2), (32, 32, 32, 4), (8, 24, 8, 2)])
def test_second_call_equals_a_fresh_network(H, W, base, levels):
    import torch
    gen = torch.Generator().manual_seed(H + W + base)
    u = torch.randn(3, H, W, generator=gen).cuda()
    t = torch.randn(3, H, W, generator=gen).cuda()

    def grads(net, k0, B):
        net.gradients(u[k0:].data_ptr(), t[k0:].data_ptr(), B)
        return net.get_grads().astype(np.float64)

    used = airt.UNet(H, W, base, levels, max_batch=3, seed=1)
    fresh = airt.UNet(H, W, base, levels, max_batch=3, seed=1)
    grads(used, 0, 3)
    got, want = grads(used, 1, 2), grads(fresh, 1, 2)
    # only the order of FP32 sums over at most 2 H W pixels differs
    assert np.linalg.norm(got - want) <= 6e-8 * 2 * H * W * np.linalg.norm(want)

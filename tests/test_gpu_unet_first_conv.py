"""Gradients for every kind of channel count of the first convolution: 1 to 8
threads per pixel, those that divide a warp and those that do not."""
import pytest

from test_gpu_unet import _check_gradients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base", [16, 24, 40, 48, 56, 64])
def test_first_convolution_widths(base):
    _check_gradients(2, base)

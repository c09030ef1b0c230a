"""Entries of matrix-free rays close to an axis against the stored matrix's.

Every ray crosses one grid line inside the image, and the image (or the
back-projected rays) has one pixel per ray, beside that crossing: a product is
a single entry.  Tolerance: the crossing's parameter is within ulps of itself
in both, so the FP64 lengths differ by a few ulps of the coordinates (1e-11 is
plenty at N = 512) and the FP32 entries by one step, 2^-23."""
import numpy as np
import pytest

from airtoolsii_b200 import testprobs as T

pytestmark = pytest.mark.gpu

N = 512


def pixels(along, line):
    """Pixel index along the ray of its crossing with `line`, and of the pixels past the line."""
    return np.floor(along) + N // 2, line + N // 2


@pytest.mark.parametrize("vertical", [False, True])
@pytest.mark.parametrize("slope", [1.5e-7, -3e-7, 1e-6, -1e-5, 1e-3])
def test_parallel(slope, vertical):
    rng = np.random.default_rng(3)
    line = np.arange(-250, 250, 3)
    along = rng.uniform(-250.0, 250.0, line.size)
    b, a = slope, np.sqrt(1.0 - slope * slope)
    if vertical:                                      # direction (b, a), normal (a, -b)
        ct, st, off = np.array([a]), np.array([-b]), a * line - b * along
    else:                                             # direction (a, b), normal (b, -a)
        ct, st, off = np.array([b]), np.array([-a]), b * along - a * line
    i, k = pixels(along, line)
    S = T.parallel_operator(N, ct, st, off)
    A = T.parallel_operator(N, ct, st, off, True)
    for side in (0, 1):                               # the pixels on both sides of the line
        ix, iy = (k - side, i) if vertical else (i, k - side)
        j = (ix * N + (N - 1 - iy)).astype(int)
        x = np.zeros(S.n)
        x[j] = 1.0
        one = np.ones(S.m)
        for want, got in ((S(x, "notransp"), A(x, "notransp")), (S(one, "transp")[j], A(one, "transp")[j])):
            assert np.count_nonzero(want) > line.size // 2
            assert np.all(np.abs(want - got) <= 2.0 ** -23 * want + 1e-11)


@pytest.mark.parametrize("slope", [1.5e-7, 1e-6, 1e-4])
def test_fan(slope):
    """Central rays through the image's middle, which they cross the axis at,
    and rays beside them."""
    w = np.arctan(slope) * np.array([-2.0, -1.0, 0.0, 1.0, 2.0])
    ct = np.array([slope, 1.0, -slope, -1.0])
    st = np.array([1.0, slope, -1.0, -slope])
    S = T.fan_operator(N, ct, st, np.cos(w), np.sin(w), 2.0 * N)
    A = T.fan_operator(N, ct, st, np.cos(w), np.sin(w), 2.0 * N, True)
    h = N // 2
    for ix, iy in ((h, h), (h - 1, h), (h, h - 1), (h - 1, h - 1), (h + 90, h), (h, h + 90), (h - 7, h - 1)):
        x = np.zeros(S.n)
        x[ix * N + N - 1 - iy] = 1.0
        want, got = S(x, "notransp"), A(x, "notransp")
        assert np.all(np.abs(want - got) <= 2.0 ** -23 * want + 1e-11)

"""Pixel-driven back projection at its edges: values that are not finite, and
detectors far wider than the image."""
import numpy as np
import pytest

from airtoolsii_b200 import testprobs as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("theta", [[17.3], [45.0], [0.0, 30.0, 90.0, 133.0]])
def test_values_that_are_not_finite_reach_their_own_pixels(theta, value):
    """As with the stored matrix: the pixels that the ray crosses, no others."""
    N = 33
    th, p, d, ct, st, off = T.parallel_tables(N, theta)
    S = T.parallel_operator(N, ct, st, off)
    A = T.parallel_operator(N, ct, st, off, True)
    rng = np.random.default_rng(0)
    for ray in rng.choice(S.m, 12, replace=False):
        u = rng.random(S.m)
        u[ray] = value
        want, got = S(u, "transp"), A(u, "transp")
        assert np.array_equal(np.isnan(want), np.isnan(got)) and np.array_equal(np.isinf(want), np.isinf(got))
        f = np.isfinite(want)
        assert np.all(np.abs(want[f] - got[f]) <= 2.0 ** -23 * np.abs(want[f]) + 1e-6)


@pytest.mark.parametrize("d", [1e7 / 3, 1e13 / 3])
@pytest.mark.parametrize("p", [7, 12])
def test_wide_detectors(p, d):
    """Offsets whose spacing rounds by more than a pixel's fraction; entries
    agree to one FP32 step and 1e-8 of their crossings."""
    N = 24
    _, p, d, ct, st, off = T.parallel_tables(N, [0.0, 20.0, 45.0, 90.0, 118.0], p, d)
    off = off + 3.3                                    # some rays through the image
    S = T.parallel_operator(N, ct, st, off)
    A = T.parallel_operator(N, ct, st, off, True)
    u = np.random.default_rng(p).random(S.m)
    a, b = S(u, "transp"), A(u, "transp")
    assert np.all(np.abs(a - b) <= 2.0 ** -23 * np.abs(a) + 1e-8)
    assert p % 2 == 0 or np.any(a > 0)


@pytest.mark.parametrize("at", [1e6, 2.0 ** 32 - 20, -(2.0 ** 32) - 9, 1e12])
def test_detectors_far_beside_the_image(at):
    """No ray meets the image, whatever its distance is in 32 bits."""
    _, _, _, ct, st, _ = T.parallel_tables(24, [0.0, 30.0, 45.0, 100.0])
    A = T.parallel_operator(24, ct, st, at + np.arange(30.0), True)
    assert not np.any(A(np.ones(A.m), "transp")) and not np.any(A(np.ones(A.n), "notransp"))


def test_two_operators_of_one_geometry_give_the_same_bits():
    """Corner pixels that several rays through the corner are corrected at."""
    N = 30
    _, p, d, ct, st, off = T.parallel_tables(N, [45.0, 45.0, 135.0, 45.0, 225.0, 45.0, 30.0, 45.0], 43)
    u = np.random.default_rng(5).uniform(-1.0, 1.0, 8 * 43)
    first = None
    for _ in range(6):
        A = T.parallel_operator(N, ct, st, off, True)
        v = A(u, "transp")
        assert first is None or np.array_equal(first, v)
        first = v

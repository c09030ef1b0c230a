"""Pixel-driven back projection of values that are not finite."""
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

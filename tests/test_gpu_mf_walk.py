"""Matrix-free operators by grid walk and pixel-driven back projection against
the stored matrix of the same geometry.

Tolerance: an entry's FP64 length differs from the traced one by a few ulps of
the coordinates, so its FP32 value by at most one FP32 step, 2^-23 relative;
a product of nonnegative vectors is then within 2^-23 of itself.  Angles next
to the axes move crossings by ulp(N)/slope, at most 1e-6 for the slopes used
here, which the absolute part covers (vectors in [0, 1])."""
import numpy as np
import pytest

import airtoolsii_b200 as airt
from airtoolsii_b200 import testprobs as T

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, 90.0, 180.0, 270.0, 45.0, 135.0, 30.0, 1e-4, 90.0001, 17.3, 61.9, 359.5]


def compare(stored, mf, seed, methods=("cimmino", "sart", "drop", "cav")):
    assert mf.matrix_free and stored.shape == mf.shape
    rng = np.random.default_rng(seed)
    x, u = rng.random(stored.n), rng.random(stored.m)
    for v, tr in ((x, "notransp"), (u, "transp")):
        a, b = stored(v, tr), mf(v, tr)
        assert np.all(np.abs(a - b) <= 2.0 ** -23 * np.abs(a) + 1e-6)
    for meth in methods:
        for a, b in zip(stored.weights(meth), mf.weights(meth)):
            np.testing.assert_allclose(b, a, rtol=1e-5)
    X = [airt.sart(A, stored(x, "notransp"), 4, None, {"lbound": 0.0})[0] for A in (stored, mf)]
    assert np.linalg.norm(X[0] - X[1]) <= 1e-5 * max(np.linalg.norm(X[0]), 1e-300)
    Y = [airt.cimmino(A, stored(x, "notransp"), 3, None, {"relaxpar": "line", "rho": 1.0})[0]
         for A in (stored, mf)]
    assert np.linalg.norm(Y[0] - Y[1]) <= 1e-5 * max(np.linalg.norm(Y[0]), 1e-300)


@pytest.mark.parametrize("N,p,d", [(2, 3, None), (31, 45, None), (32, 46, 40.0), (33, 200, 30.0),
                                   (64, 91, None), (97, 60, 130.0), (40, 57, 56.0)])
def test_parallel(N, p, d):
    th, p, d, ct, st, off = T.parallel_tables(N, SPECIAL, p, d)
    compare(T.parallel_operator(N, ct, st, off), T.parallel_operator(N, ct, st, off, True), N)


@pytest.mark.parametrize("N", [24, 65])
def test_parallel_uneven_offsets(N):
    _, p, _, ct, st, _ = T.parallel_tables(N, [3.0, 48.0, 77.7, 90.0])
    off = np.sort(np.random.default_rng(N).uniform(-0.6 * N, 0.6 * N, p))
    compare(T.parallel_operator(N, ct, st, off), T.parallel_operator(N, ct, st, off, True), N)


@pytest.mark.parametrize("N,p", [(17, 23), (32, 45), (65, 92)])
def test_fan(N, p):
    _, _, R, _, _, ct, st, cw, sw = T.fan_tables(N, SPECIAL + list(np.arange(0.0, 360.0, 24.0)), p)
    compare(T.fan_operator(N, ct, st, cw, sw, R), T.fan_operator(N, ct, st, cw, sw, R, True), N)


@pytest.mark.parametrize("N,s,p", [(16, 5, 9), (33, 33, 66), (64, 70, 31)])
def test_seismic(N, s, p):
    _, _, sx, sy, rx, ry = T.seismic_tables(N, s, p)
    compare(T.seismic_operator(N, sx, sy, rx, ry), T.seismic_operator(N, sx, sy, rx, ry, True), N)


def test_many_rays_use_fewer_parts():
    """More rays than the split into eight parts is used for."""
    th, p, d, ct, st, off = T.parallel_tables(64, np.arange(400) * 0.45 + 0.1)
    assert 400 * p > 32768
    compare(T.parallel_operator(64, ct, st, off), T.parallel_operator(64, ct, st, off, True), 1,
            methods=("sart",))

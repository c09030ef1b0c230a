"""Matrix-free solves that reach the captured iterations with the first back
projection of a new handle, nothing kept from earlier handles: they allocate
nothing there.  Tolerance: the suite's 1e-5 against the stored matrix."""
import numpy as np
import pytest

import airtoolsii_b200 as airt
from airtoolsii_b200 import testprobs as T

pytestmark = pytest.mark.gpu


def fan(mf):
    _, _, R, _, _, ct, st, cw, sw = T.fan_tables(48, np.arange(0.0, 360.0, 12.0), 60)
    return T.fan_operator(48, ct, st, cw, sw, R, mf)


def seismic(mf):
    _, _, sx, sy, rx, ry = T.seismic_tables(40, 24, 50)
    return T.seismic_operator(40, sx, sy, rx, ry, mf)


def uneven(mf):
    _, p, _, ct, st, _ = T.parallel_tables(44, [0.0, 3.0, 48.0, 77.7, 90.0, 130.0])
    off = np.sort(np.random.default_rng(2).uniform(-26.0, 26.0, p))
    return T.parallel_operator(44, ct, st, off, mf)


@pytest.mark.parametrize("method", ["cimmino", "drop"])
@pytest.mark.parametrize("make", [fan, seismic, uneven])
def test_first_back_projection_inside_the_capture(make, method):
    S = make(False)
    x = np.random.default_rng(1).random(S.n)
    b = S(x, "notransp")
    rho = 1.1                       # an upper value serves; no product runs before the solve
    want = getattr(airt, method)(S, b, [160], None, {"rho": rho, "lbound": 0.0})[0][:, -1]
    airt.release_memory()
    A = make(True)
    airt.release_memory()
    runs = [getattr(airt, method)(A, b, [160], None, {"rho": rho, "lbound": 0.0})[0][:, -1] for _ in range(2)]
    assert np.array_equal(runs[0], runs[1])
    assert np.linalg.norm(runs[0] - want) <= 1e-5 * np.linalg.norm(want)

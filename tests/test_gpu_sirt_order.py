"""The one-launch SIRT gives the launched kernels' iterates bit for bit (per-
launch profiling takes the launched ones): two, four and eight lanes per row
and column, one and several segments per group of threads, matrix in registers
and read again, bounds, tables of relaxpar and saved iterates."""
import numpy as np
import pytest
import scipy.sparse as sp

import airtoolsii_b200 as airt
from airtoolsii_b200 import _lib

pytestmark = pytest.mark.gpu


def both(A, b, method, K, opts):
    L, out = _lib.lib(), []
    for on in (1, 0):
        _lib.check(L.airt_profile_enable(A.handle, on))
        X, info = getattr(airt, method)(A, b, K, None, dict(opts))
        out.append((X, info["finaliter"]))
    return out


@pytest.mark.parametrize("N,na", [(10, 7), (24, 6), (40, 9), (64, 30), (64, 180), (100, 40), (150, 90), (200, 120)])
@pytest.mark.parametrize("method", ["cimmino", "sart"])
def test_same_bits_as_the_launched_kernels(N, na, method):
    A, b, *_ = airt.paralleltomo(N, np.linspace(0.0, 178.0, na))
    b = b + 0.02 * np.abs(b).max() * np.random.default_rng(na).standard_normal(b.size)
    assert A.nnz <= 6 << 20
    (X, _), (Y, _) = both(A, b, method, [1, 30, 300], {"rho": 1.0, "lbound": 0.0, "ubound": 1.0})
    assert np.array_equal(X, Y)
    opts = {"rho": 1.0, "relaxpar": "psi1", "stoprule": dict(type="DP", taudelta=0.2 * np.linalg.norm(b))}
    (X, i), (Y, j) = both(A, b, method, [60], opts)
    assert i == j and np.array_equal(X, Y)


@pytest.mark.parametrize("m,n,density", [(5, 400, 0.01), (400, 5, 0.5), (90000, 7, 0.3), (9, 120000, 0.4), (300, 300, 0.9)])
def test_same_bits_on_other_shapes(m, n, density):
    rng = np.random.default_rng(m)
    S = sp.random(m, n, density, "csc", random_state=n, data_rvs=lambda k: rng.uniform(0.1, 1.5, k))
    A = airt.afun_matrix(S)
    (X, _), (Y, _) = both(A, rng.random(m), "cimmino", [1, 40], {"rho": 1.0})
    assert np.array_equal(X, Y)

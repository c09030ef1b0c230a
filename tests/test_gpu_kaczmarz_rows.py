"""Kaczmarz sweeps whose steps wait on their pixels' write counts, against the
FP64 oracle: rows around the 32-entry strides and the 512 entries a warp keeps
in registers, orders that repeat rows, and the kinds of bounds.  Tolerance: the
suite's 1e-5 relative bar (the matrix is held in FP32)."""
import numpy as np
import pytest
import scipy.sparse as sp

import airtoolsii_b200 as airt
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu


def rows_matrix(lengths, n, seed):
    rng = np.random.default_rng(seed)
    ci = [np.sort(rng.choice(n, k, replace=False)) for k in lengths]
    rp = np.concatenate([[0], np.cumsum(lengths)])
    return sp.csc_matrix(sp.csr_matrix((rng.uniform(0.1, 1.0, rp[-1]), np.concatenate(ci), rp), (len(lengths), n)))


def check(method, A, sweeps, opts):
    rng = np.random.default_rng(1)
    b = A @ rng.random(A.shape[1]) + 0.01 * rng.standard_normal(A.shape[0])
    Xo, io = O.art(method, A, b, sweeps, None, opts)
    X, info = airt.art(method, airt.afun_matrix(A), b, sweeps, None, opts)
    assert X.shape == Xo.shape and info["finaliter"] == io["finaliter"]
    assert np.linalg.norm(X - Xo) <= 1e-5 * max(np.linalg.norm(Xo), 1e-300)


@pytest.mark.parametrize("lengths,n", [([1, 2, 31, 32, 33, 64, 1], 64), ([127, 128, 129, 255, 256, 257], 300),
                                       ([511, 512, 513, 700, 1, 0, 1300], 1500), ([40] * 300, 41)])
@pytest.mark.parametrize("method", ["kaczmarz", "symkaczmarz"])
def test_row_lengths(lengths, n, method):
    check(method, rows_matrix(lengths, n, n), [2, 4], {"lbound": 0.0})


def test_bounds_and_orders():
    A = rows_matrix(list(range(3, 90)), 120, 4)
    lo, hi = np.linspace(-0.5, 0.2, 120), np.linspace(0.4, 1.0, 120)
    for opts in ({}, {"lbound": 0.1, "ubound": 0.8}, {"lbound": lo, "ubound": hi}, {"ubound": hi, "damp": 0.05}):
        check("kaczmarz", A, [1, 3], opts)
    order = np.array([5, 5, 80, 2, 5, 41, 41, 0, 86, 3])
    check(order, A, [1, 3], {"lbound": lo, "relaxpar": 0.7})
    check("kaczmarz", A, [1, 3], {"relaxpar": lambda k: 1.0 / (1.0 + 0.01 * k)})

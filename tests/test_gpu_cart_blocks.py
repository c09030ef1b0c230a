"""Blocked CART sweep against the FP64 oracle at the edges of its blocks of 32
columns.  Tolerance: the existing CART bar, 1e-9 relative (the oracle runs on
the FP32-rounded matrix, so only FP64 summation order differs)."""
import numpy as np
import pytest
import scipy.sparse as sp

import airtoolsii_b200 as airt
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu


def problem(m, n, seed, density=0.2):
    rng = np.random.default_rng(seed)
    A = sp.random(m, n, density, "csc", random_state=seed, data_rvs=lambda k: rng.uniform(0.1, 1.5, k))
    A.data = A.data.astype(np.float32).astype(np.float64)
    return A, A @ rng.uniform(0.0, 1.0, n) + 0.01 * rng.standard_normal(m)


def check(A, b, K, opts, order="columnaction", x0=None):
    Xo, io = O.cart(order, A, b, K, x0, opts)
    X, info = airt.cart(order, A, b, K, x0, opts)
    assert np.linalg.norm(X - Xo) <= 1e-9 * max(np.linalg.norm(Xo), 1e-300)
    assert info["finaliter"] == io["finaliter"]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 257])
@pytest.mark.parametrize("m", [7, 90])
def test_block_edges(m, n):
    A, b = problem(m, n, 10 * n + m)
    check(A, b, [1, 2, 5], {"lbound": 0.0, "ubound": 0.9})


@pytest.mark.parametrize("n", [30, 70, 200])
def test_flags_settled_after_the_sweep(n):
    A, b = problem(60, n, n)
    x0 = np.random.default_rng(n).uniform(-2.0, 3.0, n)
    check(A, b, [2, 9], {"Kbegin": 1, "THR": 0.05, "Nunflag": 2, "seed": 5, "relaxpar": 0.6}, x0=x0)


def test_orders():
    A, b = problem(80, 150, 3)
    rng = np.random.default_rng(0)
    opts = {"Kbegin": 2, "THR": 0.02, "Nunflag": 2, "lbound": np.linspace(-1, 0, 150)}
    check(A, b, [1, 6], opts, order=rng.permutation(150))
    check(A, b, [1, 6], opts, order=rng.permutation(150)[:77])      # some columns never visited
    check(A, b, [1, 6], opts, order=np.array([4, 9, 4, 4, 140]))    # repeats: the general sweep


def test_long_columns_and_plan_reuse():
    A, b = problem(3000, 40, 8, density=0.5)                        # more entries than load ahead
    check(A, b, [3], {})
    check(A, b, [3], {}, order=np.arange(40)[::-1])                 # same matrix, another order
    check(A, b, [3], {"damp": 0.1})

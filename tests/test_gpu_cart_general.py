"""The general CART sweep (orders that repeat a column) against the FP64
oracle, with the residual in shared memory and past it.  Tolerance: the
existing CART bar, 1e-9 relative, on the FP32-rounded matrix."""
import numpy as np
import pytest
import scipy.sparse as sp

import airtoolsii_b200 as airt
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [9, 400, 26000])
def test_orders_that_repeat_a_column(m):
    rng = np.random.default_rng(m)
    n = 300
    A = sp.random(m, n, min(1.0, 40.0 / m + 0.01), "csc", random_state=m, data_rvs=lambda k: rng.uniform(0.1, 1.5, k))
    A.data = A.data.astype(np.float32).astype(np.float64)
    b = A @ rng.uniform(0.0, 1.0, n)
    order = np.concatenate([rng.permutation(n)[:200], [5, 5, 5, 299, 0, 5], rng.integers(0, n, 90)])
    opts = {"lbound": 0.0, "ubound": 0.8, "Kbegin": 2, "THR": 0.02, "Nunflag": 2, "seed": 3}
    Xo, io = O.cart(order, A, b, [1, 6], None, opts)
    X, info = airt.cart(order, A, b, [1, 6], None, opts)
    assert np.linalg.norm(X - Xo) <= 1e-9 * np.linalg.norm(Xo)
    assert info["finaliter"] == io["finaliter"]

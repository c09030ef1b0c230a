"""Schedules kept between calls belong to their very order: pairs of orders
whose FNV hashes over words are equal, one after the other on one operator.
Tolerances: the suite's bars for ART (1e-5) and CART (1e-9 on the FP32-rounded
matrix)."""
import numpy as np
import pytest
import scipy.sparse as sp

import airtoolsii_b200 as airt
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu

PAIRS = [([37923, 53913, 16485, 30457, 32727, 0], [58413, 57931, 8507, 54747, 52462, 44387]),
         ([51238, 9466, 20098, 12105, 9123, 0], [33921, 64179, 39388, 23451, 36244, 26133])]


def fnv(order):
    h = 1469598103934665603 ^ len(order)
    for j in order:
        h = ((h ^ j) * 1099511628211) % 2 ** 64
    return h


@pytest.mark.parametrize("pair", PAIRS)
def test_orders_of_equal_hash(pair):
    assert fnv(pair[0]) == fnv(pair[1])
    rng = np.random.default_rng(0)
    n, m = 1 << 16, 30
    used = sorted(pair[0] + pair[1])
    rows = np.concatenate([rng.choice(m, 7, replace=False) for _ in used])
    C = sp.csc_matrix((rng.uniform(0.2, 1.0, rows.size).astype(np.float32).astype(float),
                       (rows, np.repeat(used, 7))), shape=(m, n))
    A, At = airt.afun_matrix(C), airt.afun_matrix(C.T.tocsc())
    b, bt = rng.random(m), rng.random(n)
    for order in (pair[0], pair[1], pair[0]):
        X, _ = airt.cart(np.array(order), A, b, [3])
        Xo, _ = O.cart(np.array(order), C, b, [3])
        assert np.linalg.norm(X - Xo) <= 1e-9 * np.linalg.norm(Xo)
        X, _ = airt.art(np.array(order), At, bt, [3])
        Xo, _ = O.art(np.array(order), C.T.tocsc(), bt, [3])
        assert np.linalg.norm(X - Xo) <= 1e-5 * np.linalg.norm(Xo)

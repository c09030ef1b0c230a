"""CART where values are not finite, or nearly: a NaN or an infinity reaches
the columns that share rows with it and no others, as a column-by-column sweep
over the nonzeros gives it.  Even columns touch the rows of one half, odd ones
those of the other, so every block of columns holds both.  Tolerance: the
existing CART bar, 1e-9 relative, where the result is finite."""
import numpy as np
import pytest
import scipy.sparse as sp

import airtoolsii_b200 as airt

pytestmark = pytest.mark.gpu

M, N = 80, 75


def matrix():
    rng = np.random.default_rng(11)
    D = np.zeros((M, N))
    for j in range(N):
        rows = rng.choice(M // 2, 12, replace=False) + (M // 2 if j % 2 else 0)
        D[rows, j] = rng.uniform(0.2, 1.5, 12).astype(np.float32)
    return sp.csc_matrix(D)


def sweeps(A, b, K, x, lo, hi, lam):
    x, r = x.copy(), b.copy()
    with np.errstate(all="ignore"):
        for j in range(N):                             # r = b - A*x, nonzeros only
            q = slice(A.indptr[j], A.indptr[j + 1])
            r[A.indices[q]] -= x[j] * A.data[q]
        for _ in range(K):
            for j in range(N):
                q = slice(A.indptr[j], A.indptr[j + 1])
                rows, v = A.indices[q], A.data[q]
                od = lam * ((v @ r[rows]) / (v @ v))
                od = lo - x[j] if od < lo - x[j] else od
                od = hi - x[j] if od > hi - x[j] else od
                x[j] += od
                r[rows] -= od * v
    return x


@pytest.mark.parametrize("order", ["columnaction", "reverse"])
@pytest.mark.parametrize("what", ["nan", "inf", "-inf", "x0", "large", "diverges", "crossed", "plain"])
def test_reach_of_values_that_are_not_finite(what, order):
    A = matrix()
    rng = np.random.default_rng(1)
    b, x0, lo, hi, lam, K = A @ rng.uniform(0.0, 1.0, N), np.zeros(N), -np.inf, np.inf, 0.9, 3
    if what in ("nan", "inf", "-inf"):
        b[3] = float(what)
    elif what == "x0":
        x0[6] = np.inf
    elif what == "large":
        b[:40] *= 1e200                                # the squared norm overflows, the iterates do not
    elif what == "diverges":
        lam, K = 60.0, 12                              # overflows in the middle of a sweep
        b[:40] *= 1e250
        b[40:] = 0.0
    elif what == "crossed":
        lo, hi = 0.8, 0.2
    opts = {"relaxpar": lam, "Kbegin": 100}
    if np.isfinite(lo):
        opts.update(lbound=lo, ubound=hi)
    cols = order
    if order == "reverse":                             # the same problem with the columns turned round
        A, x0, cols = A[:, ::-1].tocsc(), x0[::-1].copy(), np.arange(N)
        A.sort_indices()
    want = sweeps(A, b, K, x0, lo, hi, lam)
    got = airt.cart(cols, A, b, [K], x0, opts)[0][:, -1]
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    f = np.isfinite(want)
    scale = np.max(np.abs(want[f]), initial=0.0)
    assert np.all(np.abs(got[f] - want[f]) <= 1e-9 * scale)
    if what in ("nan", "inf", "-inf", "x0", "diverges"):
        assert np.any(f) and not np.all(f)

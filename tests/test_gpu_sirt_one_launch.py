"""Small stored problems, whose SIRT iterations run in one launch, against the
FP64 oracle at the edges of its distribution: segments shorter and longer than
a lane group's resident vectors, empty rows and columns, more segments than
groups, both variants (with and without resident vectors), and solves longer
than one launch.  Tolerance: the suite's 1e-5 relative bar (the matrix is held
in FP32)."""
import numpy as np
import pytest
import scipy.sparse as sp

import airtoolsii_b200 as airt
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu


def random_matrix(m, n, per_row, seed, empty=0.1):
    rng = np.random.default_rng(seed)
    A = sp.random(m, n, min(1.0, per_row / n), "csr", random_state=seed, data_rvs=lambda k: rng.uniform(0.1, 1.0, k))
    keep = rng.random(m) >= empty
    return sp.csc_matrix(sp.diags(keep.astype(float)) @ A)


def check(A, K, opts, methods=("cimmino", "sart"), x0=None, seed=0):
    rng = np.random.default_rng(seed)
    b = A @ rng.random(A.shape[1]) + 0.01 * rng.standard_normal(A.shape[0])
    op = airt.afun_matrix(A)
    for meth in methods:
        o = dict(opts)
        if min(A.shape) < 3:
            o["rho"] = 1.0  # the oracle's eigs needs more unknowns
        if "stoprule" in o:
            o["stoprule"] = dict(type="DP", taudelta=o["stoprule"] * np.linalg.norm(b))
        Xo, io, _ = O.sirt(meth, A, b, K, x0, o)
        X, info = airt.sirt(meth, op, b, K, x0, dict(o, rho=io["rho"]))
        assert info["finaliter"] == io["finaliter"] and info["stoprule"] == io["stoprule"]
        assert X.shape == Xo.shape
        assert np.linalg.norm(X - Xo) <= 1e-5 * max(np.linalg.norm(Xo), 1e-300)


@pytest.mark.parametrize("m,n,per_row", [(1, 1, 1), (5, 3, 2), (40, 33, 7), (300, 700, 60), (2000, 100, 90),
                                         (64, 5000, 3000), (90000, 64, 5), (40, 90000, 9000)])
def test_shapes(m, n, per_row):
    check(random_matrix(m, n, per_row, m + n), [1, 4, 7], {"lbound": 0.0, "ubound": 1.5})


def test_larger_without_resident_vectors():
    check(random_matrix(30000, 20000, 90, 1), [2, 6], {"lbound": np.zeros(20000)}, methods=("cimmino",))


@pytest.mark.parametrize("level", [0.0, 0.3, 2.0])
def test_dp_stop_and_start_vector(level):
    A = random_matrix(400, 300, 30, 5)
    x0 = np.random.default_rng(2).random(300)
    check(A, [3, 60], {"stoprule": level, "relaxpar": "psi2"}, x0=x0)


def test_more_iterations_than_one_launch():
    A = random_matrix(60, 50, 10, 9, empty=0.0)
    check(A, [2047, 2048, 2049, 4500], {"lbound": 0.0}, methods=("sart",))

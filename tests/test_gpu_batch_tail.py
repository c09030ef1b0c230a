"""Batches whose last (or all) instances finish in one launch against the
FP64 oracle run on every instance alone: one instance, as many as the launch
takes and one more, instances that stop at different iterations and some that
never do.  Tolerance: the suite's 1e-5 relative bar, stop iterations equal."""
import numpy as np
import pytest

import airtoolsii_b200 as airt
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 7, 32, 33, 40])
@pytest.mark.parametrize("rule", ["DP", "NONE"])
def test_batch_sizes(K, rule):
    rng = np.random.default_rng(K)
    Ns = [int(rng.choice([8, 13, 16, 24])) for _ in range(K)]
    thetas = [np.sort(rng.uniform(0.0, 180.0, int(rng.integers(5, 20)))) for _ in Ns]
    B = airt.ParallelBatch(Ns, thetas)
    mats = [O.paralleltomo_matrix(N, th) for N, th in zip(Ns, thetas)]
    bs, td = [], []
    for k, (A, N) in enumerate(zip(mats, Ns)):
        b, en = airt.add_noise(A @ airt.random_ellipses(N, 5, seed=k), 0.03, seed=100 + k)
        bs.append(b)
        td.append(en * (1.05 if k % 5 else 1e-3))       # every fifth never meets the rule
    kmax = 45
    lam = np.array([1.9 / O.sirt("cimmino", A, b, [1])[1]["rho"] for A, b in zip(mats, bs)])
    xs, info = B.sirt("cimmino", bs, kmax, taudelta=td if rule == "DP" else None, relaxpar=lam, lbound=0.0)
    for k, (A, b) in enumerate(zip(mats, bs)):
        o = {"lbound": 0.0, "relaxpar": float(lam[k])}
        if rule == "DP":
            o["stoprule"] = dict(type="DP", taudelta=td[k])
        Xo, io, _ = O.sirt("cimmino", A, b, [kmax], None, o)
        assert info["finaliter"][k] == io["finaliter"] and info["stoprule"][k] == io["stoprule"]
        if io["finaliter"]:
            assert np.linalg.norm(xs[k] - Xo[:, -1]) <= 1e-5 * np.linalg.norm(Xo[:, -1])

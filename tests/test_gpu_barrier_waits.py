"""A grid barrier whose wait runs out (test hook: it waits for one arrival more
than there is, with a budget of about 1 ms): every CTA leaves, the call returns
AIRT_ERR_TIMEOUT, and the next one on the same handle gives the right result."""
import numpy as np
import pytest

import airtoolsii_b200 as airt
from airtoolsii_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture()
def stall():
    L = _lib.lib()

    def on(yes):
        assert L.airt_test_set_wait_budget(2_000_000 if yes else 4_000_000_000) == _lib.AIRT_OK
        L.airt_test_inject_stall(1 if yes else 0)
    yield on
    on(False)


def times_out(call):
    with pytest.raises(airt.AirtError) as e:
        call()
    assert e.value.code == _lib.AIRT_ERR_TIMEOUT and "bounded device wait" in str(e.value)


@pytest.mark.parametrize("N,na", [(32, 30), (200, 60)])     # matrix in registers, and read again
@pytest.mark.parametrize("rule", ["NONE", "DP"])
def test_one_launch_sirt(stall, N, na, rule):
    A, b, *_ = airt.paralleltomo(N, np.arange(na) * 180.0 / na)
    opts = {"rho": 1.0, "lbound": 0.0}
    if rule == "DP":
        opts["stoprule"] = dict(type="DP", taudelta=1e-3 * np.linalg.norm(b))
    want = airt.cimmino(A, b, [9], None, opts)[0]
    stall(True)
    times_out(lambda: airt.cimmino(A, b, [9], None, opts))
    stall(False)
    assert np.array_equal(airt.cimmino(A, b, [9], None, opts)[0], want)


def test_last_instances_of_a_batch(stall):
    B = airt.ParallelBatch([20, 32, 16], [np.arange(12) * 15.0] * 3)
    b = np.random.default_rng(0).random(B.m)
    run = lambda: B.sirt("cimmino", b, 30, relaxpar=np.ones(3))[0]  # noqa: E731
    want = run()
    stall(True)
    times_out(run)
    stall(False)
    for got, w in zip(run(), want):
        assert np.array_equal(got, w)

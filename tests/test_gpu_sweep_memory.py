"""Row and column sweeps when the device has no room for their schedules' work
space: the call goes on without it.  Allocations fail one after the other by
the host-side hook.  Tolerances: the suite's bars for ART (1e-5) and CART (1e-9
on the FP32-rounded matrix)."""
import numpy as np
import pytest

import airtoolsii_b200 as airt
from airtoolsii_b200 import _lib
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu

TH = np.arange(0.0, 180.0, 9.0)


def outcomes(solve, want, bar):
    """'ok' or 'oom' for the call whose k-th allocation fails, on a new operator each time."""
    L = _lib.lib()
    out = []
    for k in range(40):
        A = airt.paralleltomo(20, TH)[0]
        L.airt_test_fail_alloc(k)
        try:
            x = solve(A)
            assert np.linalg.norm(x - want) <= bar * np.linalg.norm(want)
            out.append("ok")
        except airt.AirtError as e:
            assert e.code == _lib.AIRT_ERR_OOM
            out.append("oom")
        finally:
            L.airt_test_fail_alloc(-1)
        assert np.linalg.norm(solve(A) - want) <= bar * np.linalg.norm(want)   # the handle stays usable
    return out


@pytest.mark.parametrize("method", ["kaczmarz", "symkaczmarz"])
def test_kaczmarz_ranks_on_the_host(method):
    M = O.paralleltomo_matrix(20, TH)
    b = M @ O.shepplogan(20)
    want = O.art(method, M, b, [4])[0][:, -1]
    out = outcomes(lambda A: getattr(airt, method)(A, b, [4])[0][:, -1], want, 1e-5)
    assert "ok" in out[:len(out) - out[::-1].index("oom")]     # one that failed before the last that must not


def test_cart_without_a_plan():
    M = O.paralleltomo_matrix(20, TH).tocsc()
    M.data = M.data.astype(np.float32).astype(np.float64)
    b = M @ O.shepplogan(20)
    want = O.cart("columnaction", M, b, [4])[0][:, -1]
    out = outcomes(lambda A: airt.columnaction(A, b, [4])[0][:, -1], want, 1e-9)
    assert "ok" in out[:len(out) - out[::-1].index("oom")]

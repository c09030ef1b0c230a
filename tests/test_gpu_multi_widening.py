"""SIRT on many right-hand sides widens part of its FP32 operands by integer
instructions (exact for finite values) and falls back to plain conversions
once an infinity or NaN is in play: both have to give the same bits."""
import numpy as np
import pytest

import airtoolsii_b200 as airt
from oracle import airt_oracle as O

pytestmark = pytest.mark.gpu


def run(op, B, X0, iters):
    import torch
    from airtoolsii_b200.batch import sirt_multi_device
    dB, dX0 = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (B, X0))
    dX = torch.empty_like(dX0)
    sirt_multi_device(op, "sart", dB.data_ptr(), dX.data_ptr(), B.shape[0], iters,
                      d_X0=dX0.data_ptr())
    return dX.cpu().numpy()


# K at the edges of the groups of 8, 16, ... 256 slots, with and without rays
# that miss (empty rows), segments of every length modulo 4
@pytest.mark.parametrize("bad", ["b", "x0"])
@pytest.mark.parametrize("N,K", [(5, 2), (16, 8), (17, 9), (24, 17), (13, 33), (20, 65), (19, 130)])
def test_nonfinite_instance_leaves_the_others_bitwise_alone(N, K, bad):
    A = O.paralleltomo_matrix(N, np.arange(0.0, 180.0, 11.0))
    op = airt.afun_matrix(A)
    rng = np.random.default_rng(K)
    # magnitudes down to the subnormal floats and up to 1e30
    scale = 10.0 ** np.linspace(-42, 30, K)[:, None]
    B = (A @ rng.random((A.shape[1], K))).T * scale
    X0 = rng.standard_normal((K, A.shape[1])) * scale
    want = run(op, B, X0, 5)
    ref = np.empty_like(want)
    for k in range(K):
        ref[k] = O.sirt("sart", A, B[k], [5], X0[k], {})[0][:, -1]
    big = scale[:, 0] >= 1e-30
    err = np.linalg.norm(want - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err[big].max() <= 1e-5
    last = K - 1
    B2, X2 = B.copy(), X0.copy()
    if bad == "b":
        B2[last, B2.shape[1] // 2] = np.nan
    else:
        X2[last, X2.shape[1] // 2] = np.inf
    got = run(op, B2, X2, 5)
    assert np.array_equal(got[:last], want[:last])
    assert not np.isfinite(got[last]).all()

"""An instance's iterates do not depend on how its solve ends: on one handle
(one choice of lanes) the instances that run on alone, in the launch for the
last ones, give the same bits as with forty running instances, which the
launched kernels take to the end.  The sizes reach all lane classes of rows
and columns, 16-bit indices included."""
import numpy as np
import pytest

import airtoolsii_b200 as airt

pytestmark = pytest.mark.gpu


def test_iterates_equal_with_and_without_the_last_launch():
    rng = np.random.default_rng(4)
    sizes = [(12, 8), (40, 20), (64, 45), (96, 70), (128, 90), (192, 60), (70, 130)]
    Ns = [sizes[k % len(sizes)][0] for k in range(40)]
    thetas = [np.sort(rng.uniform(0.0, 180.0, sizes[k % len(sizes)][1])) for k in range(40)]
    B = airt.ParallelBatch(Ns, thetas)
    b = rng.uniform(0.0, 1.0, B.m)
    td = np.full(40, 1e-12)                       # nobody stops
    full, info = B.sirt("cimmino", b, 400, taudelta=td, lbound=0.0)
    assert list(info["finaliter"]) == [400] * 40
    stay = list(range(3, 40, 4))
    td[[k for k in range(40) if k not in stay]] = 1e12
    part, info = B.sirt("cimmino", b, 400, taudelta=td, lbound=0.0)
    for k in range(40):
        assert info["finaliter"][k] == (400 if k in stay else 0)
        if k in stay:
            assert np.array_equal(full[k], part[k]), k

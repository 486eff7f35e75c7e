"""Trees of many small leaves, whose near field takes fewer threads per leaf
(32 and 64 instead of 128): the same sums as with an explicit source tile,
which always takes 128, to rounding (FP64 1e-13, mixed 2e-6: the parts of a
sum are grouped differently)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 2e-6)])
@pytest.mark.parametrize("n,ncrit,kind", [(131072, 16, "uniform"), (262144, 33, "uniform"), (60000, 2, "uniform"),
                                          (500000, 64, "uniform"), (655360, 128, "uniform"), (400000, 32, "plummer"),
                                          (300000, 64, "plummer")])
def test_threads_per_leaf_agree(n, ncrit, kind, precision, tol):
    from minimal_b200 import FMM, plummer_bodies, uniform_bodies

    xq = uniform_bodies(n, 3) if kind == "uniform" else plummer_bodies(n, 3)
    f = FMM(P=4, ncrit=ncrit, theta=0.5, precision=precision)
    f.set_bodies(xq)
    f.evaluate()
    a = f.bodies()
    f.set_tile("p2p_stage", 1536)
    f.evaluate()
    b = f.bodies()
    assert np.array_equal(a[:, :4], b[:, :4])
    assert rel(a[:, 4], b[:, 4]) < tol
    assert rel(a[:, 5:], b[:, 5:]) < tol

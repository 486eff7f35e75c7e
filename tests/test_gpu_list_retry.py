"""Lists that outgrow their first buffers: at small theta a leaf has more near
leaves and a cell more M2L entries than the sizes a new handle starts with, so
the walk is run again, after a near field and group tables made from the
dropped lists.  The first evaluation (with the retry, seen in its launches) has
the lists of the oracle and the bits of the second, whose buffers suffice, and
agrees with the oracle: FP64 within 1e-12, the mixed form within 1e-5 (FP32
pairs and split-FP16 products, and the cancellation of neutral charges), 1e-4
where its ghost sources change the order-4 truncation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


CASES = [(20000, 16, 0.25, 0), (6000, 4, 0.25, 0), (30000, 48, 0.3, 0), (3000, 16, 0.3, 1), (3000, 8, 0.25, 1)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,ncrit,theta,images", CASES)
def test_first_evaluation_after_a_retry(n, ncrit, theta, images, precision):
    import oracle
    from minimal_b200 import FMM, drand48_bodies

    xq = drand48_bodies(n, 3)
    port = oracle.Port()
    ref = port.fmm(xq, 4, ncrit, theta, images, 2 * np.pi)
    lists = port.lists()
    cells, leaves = len(port.cells()["nchild"]), int((port.cells()["nchild"] == 0).sum())
    assert len(lists["m2l_src"]) > 200 * cells + 1024 or len(lists["p2p_src"]) > 90 * leaves + 1024

    def handle():
        f = FMM(P=4, ncrit=ncrit, theta=theta, images=images, cycle=2 * np.pi, precision=precision)
        f.set_bodies(xq)
        return f

    f = handle()
    f.evaluate()
    launches = f.last_launches()
    first, own = f.bodies(), f.lists()
    for k in lists:
        assert np.array_equal(own[k], lists[k]), k
    f.evaluate()
    assert launches - f.last_launches() >= 6  # a second walk of several steps
    assert np.array_equal(f.bodies(), first)
    tol = 1e-12 if precision == "fp64" else 1e-4 if images else 1e-5
    assert np.array_equal(first[:, :4], ref[:, :4])
    assert rel(first[:, 4], ref[:, 4]) < tol
    assert rel(first[:, 5:], ref[:, 5:]) < tol

    g = handle()  # phase by phase
    for phase in (g.build_tree, g.build_lists, g.upward, g.horizontal, g.downward):
        phase()
    assert np.array_equal(g.bodies(), first)
    g.reevaluate()
    assert np.array_equal(g.bodies(), first)

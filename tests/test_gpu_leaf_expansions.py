"""P2M and L2P at every order with kernels of its own and the first without,
in both forms: multipoles and results against the oracle for leaves of one
body, of a few, and of more than a chunk (32 bodies), with bodies at the
leaf's centre and on its axis.  FP64 within 1e-12; the mixed form's multipoles
within 1e-5 per order of its largest coefficient, its results within 1e-5
(FP32 coordinates and sums, 2^-24 each, over up to 16 orders)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt((np.abs(a - b) ** 2).sum() / max((np.abs(b) ** 2).sum(), 1e-300)))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("P,n,ncrit", [(P, 600, 40) for P in range(1, 14)] +
                         [(15, 600, 40), (16, 600, 40), (17, 600, 40), (10, 2, 64), (7, 33, 64), (8, 65, 64),
                          (10, 1000, 1), (6, 5000, 200)])
def test_expansions_match_the_oracle(P, n, ncrit, precision, tol):
    import oracle
    from minimal_b200 import FMM, drand48_bodies

    xq = drand48_bodies(n, P + n)
    f = FMM(P=P, ncrit=ncrit, theta=0.4, precision=precision)
    f.set_bodies(xq)
    f.evaluate()
    port = oracle.Port()
    ref = port.fmm(xq, P, ncrit, 0.4)
    out = f.bodies()
    assert np.array_equal(out[:, :4], ref[:, :4])
    M = f.expansions()[0]
    Mr = port.expansions(P * (P + 1) // 2)[0]
    i = 0
    for order in range(P):
        a, b = M[:, i:i + order + 1], Mr[:, i:i + order + 1]
        # two opposite bodies cancel in every even order: the terms summed are
        # of size |q| r^n / n!, with r up to the leaf's corner
        terms = np.abs(xq[:, 3]).sum() / len(M) * (np.sqrt(3) * f.tree()["xr"][:, 3].min()) ** order / math.factorial(order)
        assert np.abs(a - b).max() <= tol * max(np.abs(b).max(), terms), order
        i += order + 1
    assert rel(out[:, 4], ref[:, 4]) < tol
    if n > 1:
        assert rel(out[:, 5:], ref[:, 5:]) < tol


def test_l2p_at_a_leaf_centre_and_axis():
    """Bodies at the centre of their leaf and straight above it: forces follow
    their neighbours' (a body moved by 1e-9 of the leaf)."""
    from minimal_b200 import FMM, uniform_bodies

    xq = uniform_bodies(4000, 5)
    f = FMM(P=10, ncrit=64, theta=0.4)
    f.set_bodies(xq)
    f.build_tree()
    t = f.tree()
    leaf = int(np.flatnonzero((t["nchild"] == 0) & (t["level"] == 2))[0])
    X, R = t["xr"][leaf, :3], t["xr"][leaf, 3]
    res = []
    for eps in (0.0, 1e-9):
        y = xq.copy()
        first = f.perm()[t["body"][leaf]:t["body"][leaf] + 2]
        y[first[0], :3] = X + eps * R * np.array([1, 1, 1])
        y[first[1], :3] = X + np.array([eps * R, eps * R, 0.3 * R])
        g = FMM(P=10, ncrit=64, theta=0.4)
        g.set_bodies(y)
        g.evaluate()
        o, p = g.bodies(), g.perm()
        res.append(np.stack([o[np.flatnonzero(p == b)[0]] for b in first]))
    assert np.abs(res[0][:, 4:] - res[1][:, 4:]).max() < 1e-6 * np.abs(res[1][:, 4:]).max()

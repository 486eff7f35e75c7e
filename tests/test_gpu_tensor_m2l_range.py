"""The mixed form at orders whose M2L operators exceed FP16's range unless
they are scaled: adaptive trees whose lists hold cells three and four levels
apart, uniform trees at the highest tensor-core orders, and a periodic system.
Against the FP64 form on the same tree, where the truncation is the same:
potentials of positive charges within 1e-5 of each body's own (FP32 pairs and
products of split-FP16 numbers carry about 2^-22 and add up to some 1e-6),
forces within 2e-5 of their norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bodies(n, dist, seed):
    r = np.random.default_rng(seed)
    x = (r.random((n, 3)) * 2 - 1) * np.pi
    if dist == "cluster":  # half of the bodies in balls of radius 0.03 and 0.002 inside a sparse box
        k, m = n // 2, n // 4
        x[:k] = np.array([1.1, -0.7, 0.4]) + 0.03 * (x[:k] / np.pi)
        x[:m] = np.array([-2.0, 1.9, 2.3]) + 0.002 * (x[:m] / np.pi)
    q = r.random(n) + 0.5
    return np.concatenate([x, q[:, None]], 1).astype(np.float32).astype(np.float64)


CASES = [(n, ncrit, P, theta, dist, 0)
         for n, ncrit, dist in ((6000, 16, "cluster"), (5000, 48, "uniform"))
         for P in (11, 12, 13, 14, 15) for theta in (0.4, 0.5)]
CASES += [(4000, 32, 9, 1.0, "cluster", 0), (6000, 32, 12, 0.5, "cluster", 1), (4000, 32, 13, 0.5, "uniform", 2)]


@pytest.mark.parametrize("n,ncrit,P,theta,dist,images", CASES)
def test_mixed_matches_fp64(n, ncrit, P, theta, dist, images):
    from minimal_b200 import FMM

    xq = bodies(n, dist, n + P)
    kw = dict(P=P, ncrit=ncrit, theta=theta, images=images, cycle=2 * np.pi if images else 0.0)
    out = {}
    for form in ("fp64", "mixed"):
        f = FMM(precision=form, **kw)
        f.set_bodies(xq)
        f.evaluate()
        out[form] = f.bodies()
        if form == "mixed":
            f.reevaluate()  # the kept plan
            assert np.array_equal(f.bodies(), out[form])
    a, b = out["mixed"], out["fp64"]
    assert np.array_equal(a[:, :4], b[:, :4])
    assert np.isfinite(a).all()
    assert np.abs(a[:, 4] / b[:, 4] - 1).max() < 1e-5
    assert np.sqrt(((a[:, 5:] - b[:, 5:]) ** 2).sum() / (b[:, 5:] ** 2).sum()) < 2e-5


def test_scaling_follows_theta():
    """One handle, theta changed between evaluations: the cached operators
    are those of the present scaling."""
    from minimal_b200 import FMM

    xq = bodies(6000, "cluster", 5)
    kw = dict(P=12, ncrit=16, precision="mixed")
    f = FMM(theta=0.3, **kw)
    for theta in (0.3, 0.5, 0.4):
        f.set_params(theta=theta)
        f.set_bodies(xq)
        f.evaluate()
        g = FMM(theta=theta, **kw)
        g.set_bodies(xq)
        g.evaluate()
        assert np.array_equal(f.bodies(), g.bodies())

"""The mixed form of periodic systems whose root has the largest scaled
multipole (charges of one sign, or the two signs at opposite sides): the
root's image is an M2L source of the cells on the far side, so the FP16 split
has to leave room for it.  Against the FP64 form on the same tree; the bounds
are those of FP32 pairs and split-FP16 products (about 2^-22 each, adding up
to some 1e-6): 1e-5 of the largest potential, forces 2e-5 of their norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("charges", ["positive", "sides"])
@pytest.mark.parametrize("P,theta,images", [(4, 0.5, 1), (6, 0.5, 2), (8, 0.4, 1), (10, 0.4, 3), (10, 0.5, 1)])
def test_mixed_matches_fp64(P, theta, images, charges):
    from minimal_b200 import FMM

    r = np.random.default_rng(P + images)
    n = 5003
    x = (r.random((n, 3)) * 2 - 1) * np.pi
    q = r.random(n) + 0.5
    if charges == "sides":
        q *= np.sign(x[:, 0])
    xq = np.concatenate([x, q[:, None]], 1).astype(np.float32).astype(np.float64)
    out = {}
    for form in ("fp64", "mixed"):
        f = FMM(P=P, ncrit=32, theta=theta, images=images, cycle=2 * np.pi, precision=form)
        f.set_bodies(xq)
        f.evaluate()
        out[form] = f.bodies()
    a, b = out["mixed"], out["fp64"]
    assert np.array_equal(a[:, :4], b[:, :4])
    assert np.isfinite(a).all()
    assert np.abs(a[:, 4] - b[:, 4]).max() < 1e-5 * np.abs(b[:, 4]).max()
    assert np.sqrt(((a[:, 5:] - b[:, 5:]) ** 2).sum() / (b[:, 5:] ** 2).sum()) < 2e-5


@pytest.mark.parametrize("scale", [1e-12, 1e-4, 1.0, 1e4, 1e15])
@pytest.mark.parametrize("n,P,images", [(1, 14, 2), (1, 6, 1), (1, 18, 3), (3, 12, 2)])
def test_bodies_in_one_place(n, P, images, scale):
    """A system whose root has radius 0: its local expansion, made by the
    images alone, and its near field stay in FP32's range at any period.  The images are placed
    symmetrically, so forces are zero to rounding of the potential over the
    period."""
    from minimal_b200 import FMM

    cycle = 2 * np.pi * scale
    xq = np.tile(np.float32([0.3, -0.2, 0.1, 0.75]).astype(np.float64), (n, 1))
    xq[:, :3] *= scale
    xq = xq.astype(np.float32).astype(np.float64)
    out = {}
    for form in ("fp64", "mixed"):
        f = FMM(P=P, ncrit=8, theta=0.5, images=images, cycle=cycle, precision=form)
        f.set_bodies(xq)
        f.evaluate()
        out[form] = f.bodies()
    a, b = out["mixed"], out["fp64"]
    assert np.isfinite(a).all() and np.isfinite(b).all()
    assert np.abs(a[:, 4] / b[:, 4] - 1).max() < 1e-5
    assert np.abs(a[:, 5:] - b[:, 5:]).max() < 1e-5 * np.abs(b[:, 4]).max() / cycle

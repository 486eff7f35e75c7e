"""FP64 pairs (near field and direct sums): targets among the sources,
coincident bodies in one leaf and across periodic images, and distances whose
squares are subnormal or overflow, where the sums fall back from the
normal-range pair.  Direct sums within 1e-13 of a long-double sum (a pair's
rounding, a few 2^-53, and sums of up to 3,000 terms of either sign), the
near field within 1e-12 of the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


def brute(t, s):
    d = t[:, None, :3].astype(np.longdouble) - s[None, :, :3]
    r2 = (d * d).sum(-1)
    ir = np.where(r2 > 0, 1 / np.sqrt(np.where(r2 > 0, r2, 1)), 0)
    w = s[None, :, 3] * ir
    return w.sum(1), -((w * ir * ir)[..., None] * d).sum(1)


@pytest.mark.parametrize("n,nt", [(1, 1), (31, 5), (255, 3), (257, 300), (1023, 256), (3000, 70)])
def test_direct_with_targets_among_the_sources(n, nt):
    from minimal_b200 import FMM, uniform_bodies

    xq = uniform_bodies(n, n) if n > 1 else np.array([[0.1, 0.2, 0.3, 1.0]])
    f = FMM(P=4)
    f.set_bodies(xq)
    f.build_tree()
    t = np.concatenate([xq[: (nt + 1) // 2], uniform_bodies(max(nt // 2, 1), 7)])
    out = f.direct(t)
    p, F = brute(t, xq)
    scale = np.abs(p).max() if n > 1 else 1.0
    assert np.abs(out[:, 4] - p.astype(float)).max() <= 1e-13 * max(scale, 1e-300)
    if np.abs(F).max() > 0:
        assert rel(out[:, 5:], F.astype(float)) < 1e-13


def test_direct_at_the_ends_of_the_range():
    from minimal_b200 import FMM

    xq = np.array([[0, 0, 0, 0.5], [1, 0, 0, -0.25], [0, 2, 0, 0.75]], float)
    f = FMM(P=4, ncrit=1)
    f.set_bodies(xq)
    f.build_tree()
    t = np.array([[1e-160, 0, 0, 1], [0, 1e-170, 1e-165, 1], [1e160, 0, 0, 1], [0, -3e155, 0, 1], [1e-150, 0, 0, 1],
                  [0, 0, 0, 1]])
    out = f.direct(t)
    # r2 subnormal: the potential is that of the pair; r2 infinite: nothing
    assert abs(out[0, 4] / (0.5 * (1 / np.sqrt(1e-160 * 1e-160))) - 1) < 1e-12
    assert out[1, 4] == -0.25 + 0.375 or out[1, 4] > 1e150  # r2 flushes to zero, or its inverse root
    assert np.array_equal(out[2:4, 4:], np.zeros((2, 4)))
    assert abs(out[4, 4] / 0.5e150 - 1) < 1e-12
    assert abs(out[5, 4] - (-0.25 + 0.375)) < 1e-15


@pytest.mark.parametrize("n,ncrit,images", [(40, 64, 0), (700, 64, 0), (2500, 256, 0), (2500, 7, 0), (600, 32, 1)])
def test_near_field_with_coincident_bodies(n, ncrit, images):
    import oracle
    from minimal_b200 import FMM, drand48_bodies

    cyc = 2 * np.pi
    xq = drand48_bodies(n, n, "3dp", cyc)
    xq[5:8, :3] = xq[2, :3]  # four bodies in one place
    if images:  # bodies on opposite faces: coincident across the images
        xq[10, :3] = [-np.pi, 0.5, 0.25]
        xq[11, :3] = [np.pi, 0.5, 0.25]
    f = FMM(P=6, ncrit=ncrit, theta=0.4, images=images, cycle=cyc if images else 0.0)
    f.set_bodies(xq)
    f.evaluate()
    out = f.bodies()
    ref = oracle.Port().fmm(xq, 6, ncrit, 0.4, images, cyc if images else 0.0)
    assert np.array_equal(out[:, :4], ref[:, :4])
    assert rel(out[:, 4], ref[:, 4]) < 1e-12
    assert rel(out[:, 5:], ref[:, 5:]) < 1e-12

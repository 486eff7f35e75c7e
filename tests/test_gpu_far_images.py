"""The far images of the periodic forms: eight lanes per output coefficient,
the M2L and the M2M of a sublevel in one sweep of the CTA -- orders below and
above eight (input degrees that some lanes do not have, lanes with two and
more), more outputs than the CTA has groups of lanes, one sublevel and
several.  Against the oracle, whose sums run over the same image lattice in
another order: 1e-11 covers the image shells' cancellation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("P,images", [(2, 2), (5, 3), (8, 4), (9, 2), (10, 3), (12, 6), (17, 3)])
def test_far_images_match_oracle(P, images):
    import oracle
    from minimal_b200 import FMM, drand48_bodies

    cyc = 2 * np.pi
    xq = drand48_bodies(700, P + images, "3dp", cyc)
    f = FMM(P=P, ncrit=40, theta=0.4, images=images, cycle=cyc)
    f.set_bodies(xq)
    f.evaluate()
    out = f.bodies()
    ref = oracle.Port().fmm(xq, P, 40, 0.4, images, cyc)
    assert np.array_equal(out[:, :4], ref[:, :4])
    assert rel(out[:, 4], ref[:, 4]) < 1e-11
    assert rel(out[:, 5:], ref[:, 5:]) < 1e-11

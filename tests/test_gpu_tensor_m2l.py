"""The tensor-core M2L's operand copies at every order: a multipole row is
KP / 4 chunks of 16 bytes (KP from 16 to 192) that a warp's lanes take in
sequence across rows, with the pattern compiled in (orders 4 to 12) or
counted; ranges of fewer groups than a batch of indices, and of no multiple
of it.  Against the oracle within 1e-5 (split-FP16 products and FP32 pairs
carry about 2^-22, the cancellation of neutral charges a factor of ten or so
on top), and the same bits from every evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("n,ncrit,P", [(2500, 40, P) for P in range(1, 14)] + [(130, 8, 10), (40000, 64, 10)])
def test_every_row_layout_matches_oracle(n, ncrit, P):
    import oracle
    from minimal_b200 import FMM, drand48_bodies

    xq = drand48_bodies(n, 3 * n + P)
    f = FMM(P=P, ncrit=ncrit, theta=0.5, precision="mixed")
    f.set_bodies(xq)
    f.evaluate()
    assert f.m2l_stats()["segments"] > 0
    out = f.bodies()
    ref = oracle.Port().fmm(xq, P, ncrit, 0.5)
    assert np.array_equal(out[:, :4], ref[:, :4])
    assert rel(out[:, 4], ref[:, 4]) < 1e-5
    assert rel(out[:, 5:], ref[:, 5:]) < 1e-5
    for _ in range(20):
        f.set_bodies(xq)
        f.evaluate()
        assert np.array_equal(f.bodies(), out)

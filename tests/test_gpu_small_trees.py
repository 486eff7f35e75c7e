"""Evaluations of trees too small to fill the GPU with M2L tiles, whose
contraction is split by ranges of segments between all SMs: a tile cut into
many parts, ranges of the least length, one tile with a handful of segments,
and orders on each launch shape of both contractions.  FP64 within 1e-12 of
the oracle; the mixed form within 1e-5 of it (FP32 pairs and split-FP16
products carry about 2^-22, the cancellation of neutral charges a factor of
ten or so on top)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


SHAPES = [(90, 1, 4), (300, 8, 7), (700, 32, 9), (3001, 64, 5), (3001, 16, 11), (9000, 32, 10), (20011, 64, 6),
          (20011, 64, 8), (9000, 64, 12), (5000, 32, 13)]


# (5000, 48, 14) in FP64 only: the mixed form's FP16 operators overflow at
# P = 14 (a known limit of that form, whatever the split)
@pytest.mark.parametrize("n,ncrit,P,precision,tol",
                         [s + f for f in (("fp64", 1e-12), ("mixed", 1e-5)) for s in SHAPES] +
                         [(5000, 48, 14, "fp64", 1e-12)])
def test_split_contraction_matches_oracle(n, ncrit, P, precision, tol):
    import oracle
    from minimal_b200 import FMM, drand48_bodies

    xq = drand48_bodies(n, n + P)
    f = FMM(P=P, ncrit=ncrit, theta=0.5, precision=precision)
    f.set_bodies(xq)
    f.evaluate()
    assert f.m2l_stats()["segments"] > 0
    out = f.bodies()
    ref = oracle.Port().fmm(xq, P, ncrit, 0.5)
    assert np.array_equal(out[:, :4], ref[:, :4])
    assert rel(out[:, 4], ref[:, 4]) < tol
    assert rel(out[:, 5:], ref[:, 5:]) < tol
    f.reevaluate()  # the kept plan gives the same sums
    assert np.array_equal(f.bodies(), out)

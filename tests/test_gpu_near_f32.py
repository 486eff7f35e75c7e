"""The mixed form's near field at the edges of its staging: leaves of odd and
even size (the last pair of an odd leaf is filled with a zero charge), one
leaf alone, leaves that fill a chunk, several chunks, and new charges on kept
positions.  Bodies on a jittered lattice keep every pair well separated, so
the FP32 offsets (2^-24 of the leaf radius against distances above 2^-5 of
it) leave errors below 2^-19 or 2e-6 per pair: within 5e-6 of the FP64 direct
sum plus, where leaves are split, the order-10 expansions' 1e-3 at theta 0.4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice(n, seed):
    g = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    ijk = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[g.permutation(m ** 3)[:n]]
    x = (ijk + 0.5 + g.uniform(-0.2, 0.2, (n, 3))) / m * 2 - 1
    return np.concatenate([x, g.uniform(0.5, 1.0, (n, 1))], 1)


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / max((b ** 2).sum(), 1e-300)))


def check(f, tol):
    out = f.bodies()
    t = out.copy()
    t[:, 4:] = 0
    d = f.direct(t)
    assert rel(out[:, 4], d[:, 4]) < tol
    if len(out) > 1:
        assert rel(out[:, 5:], d[:, 5:]) < tol


@pytest.mark.parametrize("n,ncrit", [(1, 64), (2, 64), (3, 64), (31, 64), (33, 64), (64, 64), (127, 256), (255, 256),
                                     (256, 256), (1001, 256), (3000, 1), (3001, 33), (20000, 256)])
def test_near_field_staging(n, ncrit):
    from minimal_b200 import FMM

    xq = lattice(n, n)
    f = FMM(P=10, ncrit=ncrit, theta=0.4, precision="mixed")
    f.set_bodies(xq)
    f.evaluate()
    tol = 5e-6 if n <= ncrit else 1e-3
    check(f, tol)
    f.set_charges(lattice(n, n + 1)[:, 3])
    f.reevaluate()
    check(f, tol)

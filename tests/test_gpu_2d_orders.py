"""The 2D passes at every order with kernels of its own and the first without,
leaf sizes on both sides of the lanes-per-leaf rule and of a warp, trees of
one leaf and of a few cells, free and periodic, against the 2D oracle:
expansions and forces within 1e-12, potentials within 1e-11 (the log potential
of far contributions cancels), as on the fixtures."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    d, n = float(np.sqrt((np.abs(a - b) ** 2).sum())), float(np.sqrt((np.abs(b) ** 2).sum()))
    return d / n if n > 0 else d


@pytest.mark.parametrize("n,P,ncrit,images", [(400, P, 8, 0) for P in range(2, 18)] +
                         [(1, 6, 8, 0), (9, 10, 8, 0), (33, 8, 1, 0), (3000, 10, 11, 0), (3000, 10, 26, 0),
                          (3001, 16, 40, 0), (2000, 9, 200, 0), (700, 10, 8, 1), (900, 13, 33, 3)])
def test_2d_matches_the_oracle(n, P, ncrit, images):
    import oracle
    from minimal_b200 import FMM

    cyc = 2 * np.pi
    g = np.random.default_rng(n * 100 + P)
    xyq = np.concatenate([g.uniform(-np.pi, np.pi, (n, 2)), g.uniform(-0.5, 0.5, (n, 1))], 1)
    if n > 20 and ncrit > 1:
        xyq[7, :2] = xyq[3, :2]  # coincident bodies
    f = FMM(P=P, ncrit=ncrit, theta=0.4, dim=2, images=images, cycle=cyc if images else 0.0)
    f.set_bodies(xyq)
    f.evaluate()
    port = oracle.Fmm2D("port")
    port.fmm(xyq, P, ncrit, 0.4, images, cyc if images else 0.0)
    out, ref = f.bodies(), port.bodies()
    assert np.array_equal(out[:, :3], ref[:, :3])
    M, L = f.expansions()
    Mr, Lr = port.expansions()
    assert rel(M, Mr) < 1e-12
    assert rel(L, Lr) < 1e-12
    assert rel(out[:, 3], ref[:, 3]) < 1e-11
    if n > 1:
        assert rel(out[:, 4:], ref[:, 4:]) < 1e-12

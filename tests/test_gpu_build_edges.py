"""Tree and lists at the sizes where the build changes its launches: body
counts around the sort's tile (2,048 keys) and its short form (32 tiles),
cell counts on both sides of it, systems of a batch around one block of first
walk steps (512 seeds).  Bit-exact against the oracle, whole numbers all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncrit", [(1, 64), (2, 1), (2047, 64), (2048, 64), (2049, 1), (4097, 8), (65535, 64),
                                     (65536, 2), (65537, 64), (70000, 1)])
def test_tree_and_lists_at_sort_edges(n, ncrit):
    import oracle
    from minimal_b200 import FMM, uniform_bodies

    xq = uniform_bodies(n, n) if n > 1 else np.array([[0.5, -0.25, 0.125, 1.0]])
    f = FMM(P=4, ncrit=ncrit, theta=0.5)
    f.set_bodies(xq)
    f.build_tree()
    f.build_lists()
    port = oracle.Port()
    port.tree(xq, ncrit)
    t, c = f.tree(), port.cells()
    for k in ("nchild", "child", "body", "nbody"):
        assert np.array_equal(t[k], c[k]), k
    assert np.array_equal(t["xr"], c["xr"])
    port.build_lists(0.5)
    la, lb = f.lists(), port.lists()
    for k in lb:
        assert np.array_equal(la[k], lb[k]), k


@pytest.mark.parametrize("nsys", [2, 64, 65, 512, 513])
def test_batch_seeds(nsys):
    from minimal_b200 import FMM, uniform_bodies

    systems = [uniform_bodies(20 + 3 * (q % 7), q) for q in range(nsys)]
    f = FMM(P=4, ncrit=4, theta=0.5)
    f.set_batch(systems)
    f.evaluate()
    out = f.bodies()
    for q in (0, nsys // 2, nsys - 1):
        g = FMM(P=4, ncrit=4, theta=0.5)
        g.set_bodies(systems[q])
        g.evaluate()
        alone, mine = g.bodies(), out[f.offsets[q]:f.offsets[q + 1]]
        assert np.array_equal(mine[:, :4], alone[:, :4])
        assert np.abs(mine[:, 4:] - alone[:, 4:]).max() <= 1e-12 * np.abs(alone[:, 4:]).max()

"""The near-field source tile on trees of many small leaves, whose default
kernels have 32 or 64 threads and tiles of their own: get_tile returns what the
kernel stages, a tile set by hand takes 128 threads until it is set back, and
the autotuner can return to the default from a tile that was set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bodies(cells, per):
    """`per` bodies in each cell of a cells^3 lattice."""
    r = np.random.default_rng(per)
    ijk = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3).repeat(per, 0)
    x = (ijk + 0.05 + 0.9 * r.random(ijk.shape)) / cells * 2 - 1
    return np.concatenate([x, r.random((len(x), 1)) + 0.5], 1).astype(np.float32).astype(np.float64)


# 32,768 leaves: of 4 bodies 32 threads, of 16 64 threads (96 and 32 leaves per
# SM are the least)
@pytest.mark.parametrize("precision,per,ncrit,want", [("fp64", 4, 8, 256), ("mixed", 4, 8, 512), ("fp64", 16, 32, 512),
                                                      ("mixed", 16, 32, 768)])
def test_tile_in_effect(precision, per, ncrit, want):
    from minimal_b200 import FMM

    xq = bodies(32, per)
    f = FMM(P=4, ncrit=ncrit, theta=0.5, precision=precision)
    default = f.get_tile("p2p_stage")
    assert default == (1536 if precision == "mixed" else 1024)
    f.set_bodies(xq)
    f.evaluate()
    assert f.get_tile("p2p_stage") == want
    out = f.bodies()
    f.set_tile("p2p_stage", 2048)
    assert f.get_tile("p2p_stage") == 2048
    f.set_tile("p2p_stage", 0)
    f.evaluate()
    assert f.get_tile("p2p_stage") == want
    assert np.array_equal(f.bodies(), out)
    f.set_bodies(xq[:500])  # another tree: few leaves
    f.evaluate()
    assert f.get_tile("p2p_stage") == default


def test_autotune_returns_to_small_leaves():
    """Leaves of four: the near field with 128 threads takes about three times
    as long (p2p.cu) and is most of an FP64 evaluation at P = 2, so the default
    wins whatever tile was set before."""
    from minimal_b200 import FMM

    f = FMM(P=2, ncrit=8, theta=0.4)
    f.set_bodies(bodies(32, 4))
    f.set_tile("p2p_stage", 2048)
    f.autotune(candidates=[8], repeats=5)
    assert f.get_tile("p2p_stage") == 256

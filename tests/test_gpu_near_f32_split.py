"""The mixed form's near field over many source leaves and chunks: against the
FP64 form on the same tree, where the truncation of the expansions is the same,
body by body.  Bodies on a jittered lattice keep every pair well separated
(FP32 errors below 2e-6 a pair, as in the single-leaf cases), and the far field
adds about 1e-6: potentials of positive charges within 1e-5 of each body's own,
forces within 1e-5 of the largest.  A source lost, doubled or given to another
leaf changes the potential of the leaves that should see it by about 1/n times
the ratio of the mean distance to its own, 2e-4 at 20,000 bodies."""
import numpy as np
import pytest

from .test_gpu_near_f32 import lattice

pytestmark = pytest.mark.gpu


# leaves of one body, odd and even ones, full ones; several chunks a leaf; the
# last two: leaves enough for 32 and 64 threads
@pytest.mark.parametrize("n,ncrit", [(1001, 256), (1500, 1), (3001, 33), (9000, 64), (20000, 256), (20011, 100),
                                     (140003, 8), (300007, 32)])
def test_split_leaves_match_fp64(n, ncrit):
    from minimal_b200 import FMM

    xq = lattice(n, n).astype(np.float32).astype(np.float64)
    q = lattice(n, n + 1)[:, 3].astype(np.float32).astype(np.float64)
    res = {}
    for form in ("fp64", "mixed"):
        f = FMM(P=6, ncrit=ncrit, theta=0.4, precision=form)
        f.set_bodies(xq)
        f.evaluate()
        res[form] = [f.bodies()]
        f.set_charges(q)
        f.reevaluate()
        res[form].append(f.bodies())
    for a, b in zip(res["mixed"], res["fp64"]):
        assert np.array_equal(a[:, :4], b[:, :4])
        assert np.abs(a[:, 4] / b[:, 4] - 1).max() < 1e-5
        assert np.abs(a[:, 5:] - b[:, 5:]).max() < 1e-5 * np.abs(b[:, 5:]).max()

"""Results written to device records on a 16-byte boundary and 8 bytes off it
(the vector and the plain kernel), 3D and 2D: the same bytes as on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(3, 1), (3, 255), (3, 4097), (2, 1), (2, 341), (2, 4097)])
def test_device_records_at_any_alignment(dim, n):
    import torch

    from minimal_b200 import FMM

    g = np.random.default_rng(n)
    f = FMM(P=4, ncrit=16, dim=dim)
    f.set_bodies(g.uniform(-1, 1, (n, dim + 1)))
    f.evaluate()
    host = f.bodies()
    buf = torch.zeros(host.size + 2, dtype=torch.float64, device="cuda")
    for off in (0, 1):
        buf.zero_()
        torch.cuda.synchronize()
        f.bodies_device(buf.data_ptr() + 8 * off)
        got = buf.cpu().numpy()
        assert np.array_equal(got[off:off + host.size].reshape(host.shape), host)
        assert not got[:off].any() and not got[off + host.size:].any()


@pytest.mark.parametrize("sizes", [[1, 1], [8192, 8193, 1], [3, 20000, 8191, 16384, 16385, 2], [1] * 700 + [9000]])
def test_uneven_batches_keep_their_roots(sizes):
    from minimal_b200 import FMM, uniform_bodies

    systems = [uniform_bodies(n, q) if n > 1 else np.array([[0.25 * q, 1.0, -2.0, 1.0]]) for q, n in enumerate(sizes)]
    f = FMM(P=4, ncrit=64, theta=0.5)
    f.set_batch(systems)
    f.evaluate()
    out = f.bodies()
    for q in {0, 1, len(sizes) // 2, len(sizes) - 1}:
        a = FMM(P=4, ncrit=64, theta=0.5)
        a.set_bodies(systems[q])
        a.evaluate()
        mine, alone = out[f.offsets[q]:f.offsets[q + 1]], a.bodies()
        assert np.array_equal(mine[:, :4], alone[:, :4])
        assert np.abs(mine[:, 4:] - alone[:, 4:]).max() <= 1e-12 * max(np.abs(alone[:, 4:]).max(), 1e-300)

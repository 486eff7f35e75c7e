"""Device memory that calls and handles give back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bodies(n, seed):
    r = np.random.default_rng(seed)
    return np.concatenate([(r.random((n, 3)) * 2 - 1) * np.pi, r.random((n, 1)) - 0.5], 1)


def free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_batch_handles_give_all_back():
    """200,000 systems have 2 MB of offsets (a quarter more with the room to
    grow): ten handles that kept theirs would hold 20 MB."""
    import torch

    from minimal_b200 import FMM

    n = 200000
    rec = torch.zeros((n, 8), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def handle():
        f = FMM(P=4, ncrit=8, theta=0.5)
        f.set_batch_device(rec.data_ptr(), np.arange(n + 1))
        f.close()

    handle()
    before = free()
    for _ in range(10):
        handle()
    assert free() >= before - (4 << 20)


@pytest.mark.parametrize("call", ["direct", "ewald"])
def test_large_target_sets_are_not_kept(call):
    """A call with many more targets than the handle has bodies works in
    memory of its own (128 and 64 bytes per target: 128 and 64 MB here); one
    with fewer stays in the handle's staging buffer, of the bodies' size."""
    from minimal_b200 import FMM

    f = FMM(P=4, ncrit=64, theta=0.5, cycle=2 * np.pi)
    f.set_bodies(bodies(1000, 2))
    f.evaluate()
    targets = bodies(1000000, 3)
    few = getattr(f, call)(targets[:64])
    getattr(f, call)(targets[:200000])
    before = free()
    many = getattr(f, call)(targets)
    assert free() >= before - (4 << 20)
    assert np.allclose(many[:64, 4:], few[:, 4:], rtol=1e-11, atol=1e-11 * np.abs(few[:, 4:]).max())

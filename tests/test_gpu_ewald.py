"""Ewald sums at sampled targets against a numpy restatement (nearest image
per axis, the integer waves of a half space, the self term): wave cutoffs from
one to many units per thread block, source counts around the tile and chunk
sizes, target counts around the targets per block, and targets that are not
bodies.  Within 1e-12 of the largest potential and of the force norm: phases
up to ksize * 2 pi carry a few 2^-53 each."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def waves_of(ksize):
    return np.array([(l, m, n) for l in range(ksize + 1) for m in range(0 if l == 0 else -ksize, ksize + 1)
                     for n in range(1 if l == 0 and m == 0 else -ksize, ksize + 1)
                     if l * l + m * m + n * n <= ksize * ksize], float)


def restated(t, b, cyc, ksize, alpha, cutoff):
    from scipy.special import erfc

    k = waves_of(ksize) * (2 * math.pi / cyc)
    k2 = (k * k).sum(1)
    fac = 8 * math.pi / cyc ** 3 * np.exp(-k2 / (4 * alpha * alpha)) / k2
    th = b[:, :3] @ k.T
    re, im = (b[:, 3] @ np.cos(th)) * fac, (b[:, 3] @ np.sin(th)) * fac
    th = t[:, :3] @ k.T
    parts = {"wave": (np.cos(th) @ re + np.sin(th) @ im, -((np.sin(th) * re - np.cos(th) * im) @ k))}
    d = t[:, None, :3] - b[None, :, :3]
    d = np.where(d < -cyc / 2, d + cyc, np.where(d > cyc / 2, d - cyc, d))
    r2 = (d * d).sum(-1)
    ok = (r2 > 0) & (r2 < cutoff * cutoff)
    r = np.sqrt(np.where(ok, r2, 1.0))
    e = np.where(ok, erfc(alpha * r) / r, 0.0)
    w = np.where(ok, (2 * alpha / math.sqrt(math.pi) * np.exp(-alpha * alpha * r * r) + e) / (r * r), 0.0)
    parts["real"] = (e @ b[:, 3], -np.einsum("ij,ijk->ik", w * b[:, 3], d))
    parts["self"] = (-2 / math.sqrt(math.pi) * alpha * t[:, 3], np.zeros((len(t), 3)))
    return parts


def close(got, want, scale_p, scale_f):
    assert np.abs(got[:, 4] - want[0]).max() <= 1e-12 * scale_p
    assert np.abs(got[:, 5:] - want[1]).max() <= 1e-12 * scale_f


@pytest.mark.parametrize("n,nt,ksize", [(1, 1, 1), (31, 3, 2), (33, 4, 7), (2000, 5, 11), (10007, 61, 9),
                                        (1025, 257, 11), (700, 9, 25)])
def test_parts_match_the_restatement(n, nt, ksize):
    from minimal_b200 import FMM

    cyc = 2.5
    g = np.random.default_rng(n + ksize)
    b = np.concatenate([g.uniform(-cyc / 2, cyc / 2, (n, 3)), g.uniform(-0.5, 0.5, (n, 1))], 1)
    t = np.concatenate([b[: (nt + 1) // 2], np.concatenate([g.uniform(-cyc / 2, cyc / 2, (nt, 3)), np.ones((nt, 1))], 1)])
    t = t[:nt]
    f = FMM(P=4, images=1, cycle=cyc)
    f.set_bodies(b)
    f.build_tree()
    alpha, cutoff = max(ksize, 3) / cyc, cyc / 2
    want = restated(t, b, cyc, ksize, alpha, cutoff)
    sp = max(np.abs(v[0]).max() for v in want.values())
    # forces are potentials times wave numbers (a body alone has none at all)
    sf = max(max(np.abs(v[1]).max() for v in want.values()), sp * 2 * math.pi * ksize / cyc)
    for name, w in want.items():
        close(f.ewald_parts(t, name, ksize=ksize, alpha=alpha, cutoff=cutoff), w, sp, sf)
    total = f.ewald(t, ksize=ksize, alpha=alpha, cutoff=cutoff)
    close(total, (sum(v[0] for v in want.values()), sum(v[1] for v in want.values())), sp, sf)
    # another wave cutoff on the same handle, then this one again
    f.ewald(t, ksize=ksize + 1, alpha=alpha, cutoff=cutoff)
    assert np.array_equal(f.ewald(t, ksize=ksize, alpha=alpha, cutoff=cutoff), total)

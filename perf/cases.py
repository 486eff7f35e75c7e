"""Performance cases: what users of the library have it compute, through its
public entry points (``minimal_b200.FMM``), and how to time one pass of each.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the inputs and the handle a program holds before the call
    run(state)          one pass; returns the results
    work(case)          bytes and flops one pass cannot do without
    exact(case, seed)   the results from plain torch in 64 bits, where affordable

Programs of the FP64 form keep 64-bit arrays and take the 64-bit Body records
as they are.  Programs of the mixed form keep 32-bit arrays: their positions
and charges are FP32 values, and they read the results back in FP32.
"""
import math

import torch

from minimal_b200 import FMM

DEV = "cuda"
CYCLE = 2 * math.pi
PAIRS_MOST = 1.2e11  # body pairs (or body-wave products) that exact() sums at most


def listed():
    return [
        # the reference drivers' own problem: 10,000 bodies from host arrays,
        # FP64, one evaluation, results back on the host
        dict(name="fp64_host_10k", kind="free", form="fp64", dist="uniform", n=10000, P=10, ncrit=64, theta=0.4,
             host=True),
        # a small particle system stepped on the device at low order, ragged
        # size: launches and latency
        dict(name="mixed_20k", kind="free", form="mixed", dist="uniform", n=20011, P=6, ncrit=64, theta=0.5,
             host=False),
        # the FP64 drop-in at scale, device-resident bodies
        dict(name="fp64_1m", kind="free", form="fp64", dist="uniform", n=1048576, P=10, ncrit=64, theta=0.4,
             host=False),
        # the headline workload: one million bodies in the mixed form
        dict(name="mixed_1m", kind="free", form="mixed", dist="uniform", n=1048576, P=10, ncrit=64, theta=0.4,
             host=False),
        # a clustered system (Plummer sphere, adaptive tree), the largest one,
        # at the leaf size the autotuner picks for it
        dict(name="plummer_4m", kind="free", form="mixed", dist="plummer", n=4194304, P=10, ncrit=96, theta=0.4,
             host=False),
        # many independent systems of uneven sizes in one evaluation
        dict(name="batch_256", kind="batch", form="mixed", nsys=256, P=6, ncrit=64, theta=0.5),
        # a periodic box with three image layers and the dipole correction:
        # mixed at scale, FP64 at an ordinary ragged size
        dict(name="periodic_mixed_1m", kind="periodic", form="mixed", n=1048576, P=10, ncrit=64, theta=0.4, images=3),
        dict(name="periodic_fp64_50k", kind="periodic", form="fp64", n=50021, P=10, ncrit=64, theta=0.4, images=3),
        # the 2D variant at its driver's size, order and leaf size
        dict(name="two_d_1m", kind="2d", form="fp64", n=1048576, P=10, ncrit=8, theta=0.4),
        # one matrix-vector product of an iterative solver: fixed positions,
        # new charges from the host, tree and lists kept
        dict(name="reevaluate_250k", kind="reevaluate", form="fp64", n=250007, P=10, ncrit=64, theta=0.4),
        # the drivers' checks of a result: direct and Ewald sums of all bodies
        # at 1,000 sampled targets
        dict(name="direct_1m", kind="direct", form="fp64", n=1048576, targets=1000),
        dict(name="ewald_1m", kind="ewald", form="fp64", n=1048576, targets=1000, ksize=11),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["free", "free", "free", "free", "batch", "periodic", "2d", "reevaluate", "direct", "ewald"])
    form = rng.choice(["fp64", "mixed"])
    P = rng.choice([4, 6, 7, 8, 9, 10, 10, 11, 12])
    ncrit = rng.choice([32, 48, 64, 64, 96, 128])
    theta = rng.choice([0.4, 0.4, 0.5])
    if kind == "free":
        dist = rng.choice(["uniform", "plummer"])
        most = 600000 if form == "fp64" else 1400000
        return dict(kind=kind, form=form, dist=dist, n=_log_int(rng, 1000, most), P=P, ncrit=ncrit, theta=theta,
                    host=rng.random() < 0.25)
    if kind == "batch":
        return dict(kind=kind, form="mixed", nsys=_log_int(rng, 4, 400), P=rng.choice([4, 6, 6, 8]), ncrit=ncrit,
                    theta=0.5)
    if kind == "periodic":
        return dict(kind=kind, form=form, n=_log_int(rng, 1000, 400000 if form == "fp64" else 1000000), P=P,
                    ncrit=ncrit, theta=theta, images=rng.choice([1, 2, 3, 3, 4]))
    if kind == "2d":
        return dict(kind=kind, form="fp64", n=_log_int(rng, 1000, 1500000), P=rng.choice([6, 8, 10, 10, 14]),
                    ncrit=rng.choice([4, 8, 8, 16, 32]), theta=theta)
    if kind == "reevaluate":
        return dict(kind=kind, form=form, n=_log_int(rng, 1000, 600000), P=P, ncrit=ncrit, theta=theta)
    return dict(kind=kind, form="fp64", n=_log_int(rng, 5000, 1048576), targets=_log_int(rng, 50, 1000),
                **(dict(ksize=rng.choice([7, 9, 11])) if kind == "ewald" else {}))


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 12345)
    return g


def _rand(shape, g):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _charges(n, g):
    q = _rand(n, g) - 0.5
    return q - q.mean()


def _bodies(case, seed):
    """N x 4 (x, y, z, q); N x 3 (x, y, q) in 2D.  Uniform in [-pi, pi]^d with
    neutral charges U[-0.5, 0.5), or a Plummer sphere (scale radius 1, radii
    up to 10) of equal charges 1/N."""
    g = _generator(seed)
    n = case["n"]
    if case.get("dist") == "plummer":
        u = 1e-12 + _rand(n, g) * ((10.0 ** 2 / (1 + 10.0 ** 2)) ** 1.5 - 1e-12)  # mass inside r <= 10
        r = 1 / torch.sqrt(u ** (-2.0 / 3.0) - 1)
        cz = 2 * _rand(n, g) - 1
        ph = 2 * math.pi * _rand(n, g)
        sz = torch.sqrt(1 - cz * cz)
        x = torch.stack([r * sz * torch.cos(ph), r * sz * torch.sin(ph), r * cz], 1)
        q = torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64)
    else:
        x = (2 * _rand((n, 2 if case["kind"] == "2d" else 3), g) - 1) * math.pi
        q = _charges(n, g)
    xq = torch.cat([x, q[:, None]], 1)
    return xq.float().double() if case["form"] == "mixed" else xq


def _sizes(case):
    """Body counts of a batch: log-uniform between 1,000 and 65,536."""
    u = torch.rand(case["nsys"], generator=torch.Generator().manual_seed(case["nsys"]), dtype=torch.float64)
    return [int(v) for v in torch.exp(math.log(1000) + u * (math.log(65536) - math.log(1000)))]


def _batch(case, seed):
    sizes = _sizes(case)
    g = _generator(seed)
    n = sum(sizes)
    xq = torch.cat([(2 * _rand((n, 3), g) - 1) * math.pi, _rand((n, 1), g) - 0.5], 1)
    return xq.float().double(), [0] + torch.tensor(sizes).cumsum(0).tolist()


def _records(xq):
    """Body records: position, charge, and room for the potential and force."""
    d = xq.shape[1] - 1
    rec = torch.zeros((len(xq), 2 * d + 2), device=xq.device, dtype=torch.float64)
    rec[:, :d + 1] = xq
    return rec


def _targets(case, xq):
    at = torch.arange(case["targets"], device=xq.device) * (len(xq) // case["targets"])
    return _records(xq[at])


def _handle(case):
    return FMM(P=case["P"], ncrit=case["ncrit"], theta=case["theta"], precision=case["form"],
               images=case.get("images", 0), cycle=CYCLE if case.get("images") else 0.0,
               dim=2 if case["kind"] == "2d" else 3)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("direct", "ewald"):
        xq = _bodies(case, seed)
        fmm = FMM(P=10, ncrit=64, theta=0.4, images=3 if kind == "ewald" else 0, cycle=CYCLE)
        rec = _records(xq)
        torch.cuda.synchronize()
        fmm.set_bodies_device(rec.data_ptr(), len(rec))
        fmm.build_tree()
        return dict(case=case, fmm=fmm, targets=_targets(case, xq).cpu().numpy())
    if kind == "batch":
        xq, offsets = _batch(case, seed)
        rec = _records(xq)
        return dict(case=case, fmm=_handle(case), rec=rec, out=torch.empty_like(rec), offsets=offsets)
    xq = _bodies(case, seed)
    if case.get("host"):
        return dict(case=case, fmm=_handle(case), xq=xq.cpu().numpy())
    rec = _records(xq)
    state = dict(case=case, fmm=_handle(case), rec=rec, out=torch.empty_like(rec))
    if kind == "reevaluate":
        torch.cuda.synchronize()
        state["fmm"].set_bodies_device(rec.data_ptr(), len(rec))
        state["fmm"].evaluate()
        state["q"] = _new_charges(case, seed).cpu().numpy()
    return state


def _new_charges(case, seed):
    q = _charges(case["n"], _generator(int(seed) + 1000003))
    return q.float().double() if case["form"] == "mixed" else q


# ---------------------------------------------------------------- one pass
def run(state):
    case, fmm = state["case"], state["fmm"]
    kind = case["kind"]
    if kind == "direct":
        t = fmm.direct(state["targets"])
        return {"p": t[:, 4], "F": t[:, 5:]}
    if kind == "ewald":
        t = fmm.ewald(state["targets"], ksize=case["ksize"])
        return {"p": t[:, 4], "F": t[:, 5:]}
    if case.get("host"):
        fmm.set_bodies(state["xq"])
        fmm.evaluate()
        out = fmm.bodies()
        if case["form"] == "mixed":
            out = out.astype("float32")
        return _parts(out, 3)
    rec, out = state["rec"], state["out"]
    # the handle works on its own stream: torch's last work on these buffers
    # (the FP32 results below) has to be over
    torch.cuda.current_stream().synchronize()
    if kind == "reevaluate":
        fmm.set_charges(state["q"])
        fmm.reevaluate()
    else:
        if kind == "batch":
            fmm.set_batch_device(rec.data_ptr(), state["offsets"])
        else:
            fmm.set_bodies_device(rec.data_ptr(), len(rec))
        fmm.evaluate()
        if kind == "periodic":
            fmm.dipole_correction()
    fmm.bodies_device(out.data_ptr())
    if case["form"] == "mixed":
        out = out.float()
    return _parts(out, 2 if kind == "2d" else 3)


def _parts(out, d):
    return {"Xq": out[:, :d + 1], "p": out[:, d + 1], "F": out[:, d + 2:]}


# ---------------------------------------------------------------- work
def work(case):
    """Body records' X and q read and whole records written once; the flops of
    the near field (20 per body pair in 3D, 16 in 2D with one logarithm counted
    as one) and of the multipole-to-local translations, from the list lengths
    of a uniform tree at theta = 0.4: 74 near leaves of a leaf and 173 (2D: 25
    and 60) translations per cell, fewer at a larger theta.  Direct and Ewald
    sums: the pairs, 20 flops each (Ewald: the half that lies within the
    cutoff sphere at 60) plus 20 flops per body and wave."""
    kind = case["kind"]
    if kind in ("direct", "ewald"):
        n, t = case["n"], case["targets"]
        if kind == "direct":
            return {"bytes": 32 * n + 96 * t, "flops": 20 * n * t}
        waves = 2 / 3 * math.pi * case["ksize"] ** 3
        return {"bytes": 32 * n + 96 * t, "flops": 30 * n * t + 20 * waves * (n + t)}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for n in _sizes(case):
            w = work(dict(case, kind="free", n=n))
            total = {key: total[key] + w[key] for key in total}
        return total
    n, P = case["n"], case["P"]
    d = 2 if kind == "2d" else 3
    if case.get("dist") == "plummer":
        m = 0.3 * case["ncrit"]
    else:
        m = n / (2 ** d) ** max(0, math.ceil(math.log(max(1.0, n / case["ncrit"])) / math.log(2 ** d)))
    shrink = (0.4 / case["theta"]) ** d
    cells = n / m * 2 ** d / (2 ** d - 1)
    near, far = (25, 60) if d == 2 else (74, 173)
    near, far = min(n, near * shrink * m), min(cells, far * shrink)
    if d == 2:
        flops = 16 * near * n + 8 * P * P * far * cells
    else:
        blocks = sum((j + 1) * (k + 1) for j in range(P) for k in range(P - j))
        flops = 20 * near * n + 8 * blocks * far * cells
    record = 8 * (2 * d + 2)
    read = 8 * n if kind == "reevaluate" else 8 * (d + 1) * n
    return {"bytes": read + record * n, "flops": flops}


# ---------------------------------------------------------------- 64-bit results
def _tree_order(x, ncrit):
    """Body order of the octree: octants in digit order (a coordinate above its
    cell's centre sets its bit; x lowest), bodies of one leaf (at most ncrit)
    in input order.  Root: the bounds' centre and 1.00001 of the largest
    half-extent."""
    lo, hi = x.min(0).values, x.max(0).values
    c = ((hi + lo) / 2).expand_as(x).clone()
    r = max(float((c[0] - lo).max()), float((hi - c[0]).max())) * 1.00001
    levels = 21
    key = torch.zeros(len(x), dtype=torch.int64, device=x.device)
    leaf = torch.zeros_like(key)
    todo = torch.ones(len(x), dtype=torch.bool, device=x.device)
    for level in range(levels + 1):
        _, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
        done = todo & (cnt[inv] <= ncrit)
        leaf[done] = key[done] << (3 * (levels - level))
        todo &= ~done
        if not bool(todo.any()) or level == levels:
            break
        up = x > c
        for d in range(x.shape[1]):
            key = key + (up[:, d].long() << d) if d else key * 8 + up[:, 0].long()
        r *= 0.5
        c = c + torch.where(up, r, -r)
    return torch.sort(leaf, stable=True).indices


def _direct(t, x, q):
    """Potential and force of bodies (x, q) at points t, in 64 bits: the 1/r
    kernel in 3D, log(1/r) in 2D."""
    d = x.shape[1]
    p = torch.zeros(len(t), dtype=torch.float64, device=x.device)
    f = torch.zeros_like(t)
    step = max(1, (1 << 25) // len(x))
    for a in range(0, len(t), step):
        dx = [t[a:a + step, k, None] - x[None, :, k] for k in range(d)]
        r2 = sum(v * v for v in dx)
        r2 = torch.where(r2 == 0, math.inf, r2)
        if d == 3:
            w = 1 / torch.sqrt(r2)
            p[a:a + step] = w @ q
            w = w / r2
        else:
            w = 1 / r2
            p[a:a + step] = torch.where(w > 0, -0.5 * torch.log(torch.where(w > 0, r2, 1.0)), 0.0) @ q
        for k in range(d):
            f[a:a + step, k] = -(dx[k] * w) @ q
    return p, f


def _wave_vectors(ksize):
    """The half space of integer wave vectors with 0 < |k| <= ksize."""
    k = torch.arange(-ksize, ksize + 1, device=DEV)
    l, m, n = (v.reshape(-1) for v in torch.meshgrid(k, k, k, indexing="ij"))
    half = (l > 0) | ((l == 0) & (m > 0)) | ((l == 0) & (m == 0) & (n > 0))
    keep = half & (l * l + m * m + n * n <= ksize * ksize)
    return torch.stack([l, m, n], 1)[keep].double()


def _ewald(t, qt, x, q, ksize, alpha, cutoff):
    """Ewald sum (conducting boundary) of bodies (x, q) at points t with
    charges qt: the nearest image per axis within the cutoff, the waves up to
    ksize, and the self term."""
    k = _wave_vectors(ksize) * (2 * math.pi / CYCLE)
    k2 = (k * k).sum(1)
    fac = 8 * math.pi / CYCLE ** 3 * torch.exp(-k2 / (4 * alpha * alpha)) / k2
    re, im = torch.zeros_like(k2), torch.zeros_like(k2)
    step = max(1, (1 << 24) // len(k))
    for a in range(0, len(x), step):
        th = x[a:a + step] @ k.T
        re += q[a:a + step] @ torch.cos(th)
        im += q[a:a + step] @ torch.sin(th)
    re, im = re * fac, im * fac
    p, f = torch.zeros(len(t), dtype=torch.float64, device=x.device), torch.zeros_like(t)
    for a in range(0, len(t), step):
        th = t[a:a + step] @ k.T
        c, s = torch.cos(th), torch.sin(th)
        p[a:a + step] = c @ re + s @ im
        f[a:a + step] = -(s * re - c * im) @ k
    step = max(1, (1 << 25) // len(x))
    for a in range(0, len(t), step):
        dx = [t[a:a + step, d, None] - x[None, :, d] for d in range(3)]
        dx = [torch.where(v.abs() > CYCLE / 2, v - torch.sign(v) * CYCLE, v) for v in dx]
        r2 = sum(v * v for v in dx)
        r2 = torch.where((r2 > 0) & (r2 < cutoff * cutoff), r2, math.inf)
        r = torch.sqrt(r2)
        e = torch.erfc(alpha * r) / r
        w = (2 * alpha / math.sqrt(math.pi) * torch.exp(-alpha * alpha * r2) + e) / r2
        w, e = torch.where(torch.isinf(r), 0.0, w), torch.where(torch.isinf(r), 0.0, e)
        p[a:a + step] += e @ q
        for d in range(3):
            f[a:a + step, d] -= (dx[d] * w) @ q
    return p - 2 * alpha / math.sqrt(math.pi) * qt, f


def exact(case, seed):
    kind = case["kind"]
    if kind in ("direct", "ewald"):
        xq = _bodies(case, seed)
        x, q = xq[:, :3].contiguous(), xq[:, 3].contiguous()
        t = _targets(case, xq)[:, :4]
        if kind == "direct":
            p, f = _direct(t[:, :3].contiguous(), x, q)
        else:
            p, f = _ewald(t[:, :3].contiguous(), t[:, 3], x, q, case["ksize"], case["ksize"] / CYCLE, CYCLE / 2)
        return {"p": p, "F": f}
    if kind == "batch":
        sizes = _sizes(case)
        if sum(v * v for v in sizes) > PAIRS_MOST:
            return None
        xq, offsets = _batch(case, seed)
        parts = [_free_space(case, xq[a:b]) for a, b in zip(offsets, offsets[1:])]
        return {k: torch.cat([v[k] for v in parts]) for k in parts[0]}
    if case["n"] ** 2 > (PAIRS_MOST / 10 if kind == "periodic" else PAIRS_MOST):
        return None
    xq = _bodies(case, seed)
    if kind == "reevaluate":
        xq[:, -1] = _new_charges(case, seed)
    return _periodic(case, xq) if kind == "periodic" else _free_space(case, xq)


def _free_space(case, xq):
    d = xq.shape[1] - 1
    xq = xq[_tree_order(xq[:, :d], case["ncrit"])]
    x, q = xq[:, :d].contiguous(), xq[:, d].contiguous()
    p, f = _direct(x, x, q)
    return {"Xq": xq, "p": p, "F": f}


def _periodic(case, xq):
    """Forces of the infinite periodic system with a conducting boundary,
    which the finite cube of images approaches once its dipole term is taken
    off.  The images' potential differs from it by that term (and one image
    layer alone by more), so it has no such value."""
    xq = xq[_tree_order(xq[:, :3], case["ncrit"])]
    x, q = xq[:, :3].contiguous(), xq[:, 3].contiguous()
    f = _ewald(x, q, x, q, 24, 2.0, CYCLE / 2)[1] if case["images"] >= 3 else None
    return {"Xq": xq, "p": None, "F": f}

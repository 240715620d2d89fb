"""The work that users of this framework have it do, as cases that can be timed.

Every case calls the package's public entry points as a program does: one-shot transforms,
plans replayed with new amplitudes and phases, the object -> projector -> projection chain,
a gradient step of a phase-only hologram, a batch of uneven problems, the Monte Carlo
estimator, and the FP64 mode that is the default of the `holo` executable and of the
reference's own names.  Geometry: objects of 10 um pitch 0.2 to 0.5 m above a projector of
7.56 um pitch, or rings of points as the executable generates by default.

The split32 mode carries about six digits, so the programs here keep its fields in complex64
(and, in a gradient step, the phases in float32, whose gradients then come back in float32);
FP64 fields stay complex128.
"""
import math

import numpy as np
import torch

import __graft_entry__

holo = __graft_entry__.load_package()

DEV = "cuda:0"
PITCH_OBJECT, PITCH_PROJECTOR = 10e-6, 7.56e-6
LAMBDAS = (632.8e-9, 650e-9)


def listed():
    return [
        # the executable's smallest use: a ring of points onto a small projector, the
        # reference's own function on NumPy arrays in FP64 (host buffers in and out)
        dict(name="ring_fp64_host", kind="reference_call", n=256, m=16384, dist=0.35, lam=650e-9,
             layout="ring", offset=0.0, sign=-1),
        # a ragged number of object points onto the default 512^2 projector in FP64
        dict(name="object_fp64", kind="transform", precision="fp64", n=1000, m=262144, dist=0.25,
             lam=650e-9, layout="lattice", offset=0.0, sign=-1),
        # the whole FP64 chain of a small hologram
        dict(name="chain64_fp64", kind="chain", precision="fp64", n=4096, m=65536, p=4096,
             dist=0.35, lam=632.8e-9, layout="lattice", offset=0.0),
        # the smallest replay: launches and latency (an interactive preview)
        dict(name="replay_small", kind="replay", n=1024, m=4096, dist=0.35, lam=632.8e-9,
             layout="lattice", offset=0.0, sign=-1),
        # a plan replayed with new phases, projector at display size
        dict(name="replay_display", kind="replay", n=16384, m=262144, dist=0.3, lam=632.8e-9,
             layout="lattice", offset=0.0, sign=-1),
        # one call with new positions, ragged counts, jittered points, off the axis
        dict(name="ragged_oneshot", kind="transform", precision="split32", n=10007, m=50021,
             dist=0.41, lam=650e-9, layout="jitter", offset=0.7e-3, sign=1),
        # the chain of a small hologram, planning included
        dict(name="chain64", kind="chain", precision="split32", n=4096, m=65536, p=4096, dist=0.35,
             lam=632.8e-9, layout="lattice", offset=0.0),
        # the benchmark's chain: 512^2 object, 1024^2 projector, 512^2 projection
        dict(name="chain512", kind="chain", precision="split32", n=262144, m=1048576, p=262144,
             dist=0.35, lam=632.8e-9, layout="lattice", offset=0.0),
        # one gradient step of a phase-only hologram, small and at full size
        dict(name="step256", kind="step", n=65536, m=65536, dist=0.35, lam=632.8e-9,
             layout="lattice", offset=0.0),
        dict(name="step1024", kind="step", n=1048576, m=262144, dist=0.35, lam=632.8e-9,
             layout="lattice", offset=0.0),
        # 64 uneven holograms in one batched launch
        dict(name="batch64", kind="batch", count=64, most=262144, side=1024, lam=632.8e-9),
        # one in sixteen sources per block of 256 targets
        dict(name="mc16", kind="mc", n=4096, m=65536, dist=0.35, lam=632.8e-9, layout="lattice",
             offset=0.0, sign=-1, subsample=16, block=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, n_range, m_range, most):
    """Two sizes over their ranges' logarithms, half of them odd ones, at most `most` pairs."""
    while True:
        n, m = _log(rng, *n_range), _log(rng, *m_range)
        if rng.random() < 0.5:  # square planes
            n, m = max(1, round(math.sqrt(n))) ** 2, max(1, round(math.sqrt(m))) ** 2
        if n * m <= most:
            return n, m


def draw(rng):
    kind = rng.choice(["reference_call", "transform", "transform", "replay", "replay", "chain",
                       "chain", "step", "batch", "mc"])
    case = dict(kind=kind, lam=rng.choice(LAMBDAS))
    if kind == "batch":
        case.update(count=rng.randint(3, 48), most=_log(rng, 4096, 262144),
                    side=rng.choice([256, 512, 768, 1024]))
        return case
    case.update(dist=rng.uniform(0.2, 0.5), layout=rng.choice(["lattice", "lattice", "jitter"]),
                offset=rng.choice([0.0, rng.uniform(0.0, 1e-3)]))
    if kind == "reference_call":
        n, m = _sizes(rng, (1, 2000), (1024, 262144), 1e8)
        case.update(n=n, m=m, layout=rng.choice(["ring", "lattice"]), sign=rng.choice([-1, 1]))
    elif kind == "transform":
        precision = rng.choice(["split32", "split32", "fp64"])
        n, m = (_sizes(rng, (64, 16384), (1024, 262144), 1e9) if precision == "fp64" else
                _sizes(rng, (64, 262144), (1024, 1048576), 1e11))
        case.update(precision=precision, n=n, m=m, sign=rng.choice([-1, 1]))
    elif kind == "replay":
        n, m = _sizes(rng, (256, 262144), (1024, 1048576), 1e11)
        case.update(n=n, m=m, sign=rng.choice([-1, 1]))
    elif kind == "chain":
        precision = rng.choice(["split32", "split32", "fp64"])
        most = 3e8 if precision == "fp64" else 1e11
        n, m = _sizes(rng, (256, 262144), (4096, 1048576), most)
        case.update(precision=precision, n=n, m=m, p=_sizes(rng, (256, 262144), (m, m), most)[0])
    elif kind == "step":
        n, m = _sizes(rng, (4096, 1048576), (1024, 262144), 1e11)
        case.update(n=n, m=m)
    else:
        n, m = _sizes(rng, (1024, 65536), (4096, 262144), 4e9)
        case.update(n=n, m=m, sign=rng.choice([-1, 1]), subsample=rng.choice([4, 16, 25]),
                    block=rng.choice([256, 512, 1024]))
    return case


# ---- inputs -----------------------------------------------------------------------------
def _plane(count, pitch, z, dx=0.0):
    """The first `count` points of a centred square lattice at height z (count x 3)."""
    side = math.ceil(math.sqrt(count))
    i = torch.arange(count, device=DEV)
    c = (side - 1) / 2.0
    x = (torch.div(i, side, rounding_mode="floor").double() - c) * pitch + dx
    y = ((i % side).double() - c) * pitch
    return torch.stack([x, y, torch.full_like(x, z)], dim=1)


def _object(case, gen):
    if case["layout"] == "ring":  # a circle 1 mm wide, as the executable generates
        t = torch.arange(case["n"], device=DEV).double() * (2 * math.pi / case["n"])
        return torch.stack([torch.sin(t) * 0.5e-3, torch.cos(t) * 0.5e-3,
                            torch.full_like(t, case["dist"])], dim=1)
    u = _plane(case["n"], PITCH_OBJECT, case["dist"], case["offset"])
    if case["layout"] == "jitter":
        u[:, :2] += (_uniform(gen, (case["n"], 2)) - 0.5) * PITCH_OBJECT
    return u


def _uniform(gen, shape):
    return torch.rand(shape, generator=gen, dtype=torch.float64, device=DEV)


def _blobs(gen, count):
    """Eight Gaussian blobs on a square image, its first `count` pixels, in (0, 1]."""
    side = math.ceil(math.sqrt(count))
    c = torch.arange(side, device=DEV).double()
    img = torch.zeros(side, side, dtype=torch.float64, device=DEV)
    for cx, cy, s, peak in _uniform(gen, (8, 4)).tolist():
        s = side * (0.01 + 0.07 * s)
        img += (0.2 + 0.8 * peak) * (torch.exp(-(c - cx * side) ** 2 / (2 * s * s))[:, None] *
                                     torch.exp(-(c - cy * side) ** 2 / (2 * s * s))[None, :])
    return (img / img.max()).reshape(-1)[:count].contiguous()


class _Inputs:
    """What a program holds before the call; a plan or batch goes with it."""

    plan = batch = None

    def __init__(self, **fields):
        self.__dict__.update(fields)

    def __del__(self):
        for kept in (self.plan, self.batch):
            if kept is not None:
                kept.close()


def _inputs(case, seed):
    """The inputs alone: positions, amplitudes and phases (no plan, no call of the package)."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    tau = 2 * math.pi
    if case["kind"] == "batch":
        rng = np.random.default_rng(seed)
        shapes = np.random.default_rng(case["count"] * 7919 + case["most"])  # the case's own sizes
        problems = []
        for _ in range(case["count"]):
            n = int(np.exp(shapes.uniform(np.log(1024), np.log(case["most"]))))
            m = int(shapes.choice([s for s in (128, 256, 512, 768, 1024) if s <= case["side"]])) ** 2
            problems.append((_uniform(gen, n), _uniform(gen, n) * tau,
                             _plane(n, PITCH_OBJECT, rng.uniform(0.2, 0.5)),
                             _plane(m, PITCH_PROJECTOR, 0.0)))
        return _Inputs(problems=problems, case=case)
    if case["kind"] == "step":  # projector pixels at z = 0 onto a target image
        return _Inputs(case=case, u=_plane(case["n"], PITCH_PROJECTOR, 0.0),
                       v=_object(dict(case, n=case["m"]), gen),
                       phase=(_uniform(gen, case["n"]) * tau).float(),
                       amp=torch.ones(case["n"], dtype=torch.float64, device=DEV),
                       target=_unit_mean(_blobs(gen, case["m"])))
    u, v = _object(case, gen), _plane(case["m"], PITCH_PROJECTOR, 0.0)
    chain = case["kind"] == "chain"
    s = _Inputs(case=case, u=u, v=v, phase=_uniform(gen, case["n"]) * tau,
                amp=_blobs(gen, case["n"]) if chain else _uniform(gen, case["n"]))
    if chain:
        s.w = _plane(case["p"], PITCH_OBJECT, case["dist"], case["offset"])
    return s


def _unit_mean(image):
    return image / image.mean()


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        # one buffer holds every problem's field, each problem writes its part
        s.field = torch.zeros(sum(2 * v.shape[0] for *_, v in s.problems), dtype=torch.float64,
                              device=DEV)
        todo, at = [], 0
        for amp, phase, u, v in s.problems:
            y = s.field[at:at + 2 * v.shape[0]]
            at += 2 * v.shape[0]
            todo.append(holo.Problem(amp, phase, u.reshape(-1), v.reshape(-1), -1, case["lam"], y))
        s.batch = holo.Batch(todo, "split32")
        return s
    if kind == "reference_call":
        x = torch.stack([s.amp, s.phase], dim=1)
        s.x, s.u, s.v = (t.cpu().numpy() for t in (x, s.u, s.v))
        return s
    s.u, s.v = s.u.reshape(-1), s.v.reshape(-1)
    if kind == "chain":
        s.w = s.w.reshape(-1)
    if kind in ("replay", "step"):
        s.plan = holo.Plan(s.u, s.v, "split32")
    return s


def run(s):
    case = s.case
    kind, lam = case["kind"], case["lam"]
    if kind == "reference_call":
        return holo.transform_full(s.x, s.u, s.v, case["sign"], lam)
    if kind == "transform":
        y = holo.transform(s.amp, s.phase, s.u, s.v, case["sign"], lam, precision=case["precision"])
        return y if case["precision"] == "fp64" else y.to(torch.complex64)
    if kind == "replay":
        return s.plan.execute(s.amp, s.phase, case["sign"], lam).to(torch.complex64)
    if kind == "chain":
        ya, yp, za, zp = holo.project(s.amp, s.phase, s.u, s.v, s.w, lam,
                                      precision=case["precision"])
        if case["precision"] == "fp64":
            return ya, yp, za, zp
        return torch.polar(ya.float(), yp.float()), torch.polar(za.float(), zp.float())
    if kind == "step":
        from holo_gb300 import torch_ops
        phase = s.phase.detach().requires_grad_(True)
        z = torch_ops.huygens(s.amp, phase, s.plan, +1, lam)
        torch_ops.intensity_loss(z, s.target).backward()
        return z.detach().float(), phase.grad
    if kind == "batch":
        s.batch.execute()
        return s.field.float()
    return holo.transform_mc(s.amp, s.phase, s.u, s.v, case["sign"], lam, seed=7,
                             subsample=case["subsample"],
                             targets_per_block=case["block"]).to(torch.complex64)


# ---- what a pass cannot do without --------------------------------------------------------
FLOP_PER_PAIR = 29  # the reference's count for one source-target term in FP64


def _batch_sizes(case):
    shapes = np.random.default_rng(case["count"] * 7919 + case["most"])
    for _ in range(case["count"]):
        n = int(np.exp(shapes.uniform(np.log(1024), np.log(case["most"]))))
        yield n, int(shapes.choice([s for s in (128, 256, 512, 768, 1024) if s <= case["side"]])) ** 2


def work(case):
    """Bytes: positions, amplitudes and phases in, fields (or gradients) out, once each.

    Flops: an FP64 result holds the rounding of every distance, so each pair has to be
    formed; a split32 result does not (smooth sums can be regrouped), which leaves the
    work per point: a distance, a sine and a cosine, about as much as one pair."""
    kind = case["kind"]
    if kind == "batch":
        points = [(n, m) for n, m in _batch_sizes(case)]
        # positions are held by the batch: amplitudes and phases in, fields out
        return {"bytes": sum(16 * n + 16 * m for n, m in points),
                "flops": FLOP_PER_PAIR * sum(n + m for n, m in points)}
    n, m = case["n"], case["m"]
    fp64 = kind == "reference_call" or case.get("precision") == "fp64"
    if kind == "chain":
        p = case["p"]
        return {"bytes": 40 * n + 40 * m + 40 * p,
                "flops": FLOP_PER_PAIR * (m * (n + p) if fp64 else n + 2 * m + p)}
    if kind == "step":
        return {"bytes": 4 * n + 4 * n + 8 * n + 16 * m, "flops": FLOP_PER_PAIR * 2 * (n + m)}
    held = kind == "replay"
    return {"bytes": (16 if held else 40) * n + (16 if held else 40) * m,
            "flops": FLOP_PER_PAIR * (n * m if fp64 else n + m)}


# ---- the same in plain 64-bit torch -------------------------------------------------------
MOST_PAIRS = 1.2e10  # above this the 64-bit sum takes too long


def _sum64(amp, phase, u, v, sign, lam):
    """y_m = sum_n a_n exp(i (phi_n + sign k r_nm)) / r_nm in float64."""
    k = (2.0 * math.pi) / lam
    y = torch.empty(v.shape[0], dtype=torch.complex128, device=DEV)
    step = max(1, (1 << 24) // max(1, u.shape[0]))
    for at in range(0, v.shape[0], step):
        t = v[at:at + step]
        d = [t[:, None, i] - u[None, :, i] for i in range(3)]
        r = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        kr = r * k
        ph = phase[None, :] + kr if sign > 0 else phase[None, :] - kr
        w = amp[None, :] / r
        y[at:at + step] = torch.complex((w * torch.cos(ph)).sum(1), (w * torch.sin(ph)).sum(1))
    return y


def _polar64(y):
    top = y.abs().max()
    if top >= 1e-6:
        y = y / top
    return y.abs(), torch.angle(y)


def exact(case, seed):
    kind, lam = case["kind"], case["lam"]
    if kind == "mc":
        return None  # which sources a block picks is the estimator's own
    if kind == "batch":
        pairs = sum(n * m for n, m in _batch_sizes(case))
    else:
        pairs = case["n"] * case["m"]
        pairs += case["m"] * case["p"] if kind == "chain" else pairs if kind == "step" else 0
    if pairs > MOST_PAIRS:
        return None
    s = _inputs(case, seed)
    if kind == "batch":
        return torch.cat([torch.view_as_real(_sum64(a, ph, u, v, -1, lam)).reshape(-1)
                          for a, ph, u, v in s.problems])
    if kind == "chain":
        ya, yp = _polar64(_sum64(s.amp, s.phase, s.u, s.v, -1, lam))
        za, zp = _polar64(_sum64(ya, yp, s.v, s.w, +1, lam))
        if case["precision"] == "fp64":
            return ya, yp, za, zp
        return torch.polar(ya, yp), torch.polar(za, zp)
    if kind == "step":
        phase = s.phase.double()
        z = torch.view_as_real(_sum64(s.amp, phase, s.u, s.v, +1, lam)).requires_grad_(True)
        inten = z[:, 0] ** 2 + z[:, 1] ** 2
        torch.mean((inten / inten.mean() - s.target) ** 2).backward()
        g = torch.view_as_complex(z.grad)
        # dL/dphi_n = -a_n Im(e^{i phi_n} conj(sum_m G_m e^{-i k r_nm} / r_nm))
        h = _sum64(g.abs(), torch.angle(g), s.v, s.u, -1, lam)
        wave = torch.polar(torch.ones_like(phase), phase) * h.conj()
        return z.detach(), -s.amp * wave.imag
    y = _sum64(s.amp, s.phase, s.u, s.v, case["sign"], lam)
    return y.cpu().numpy() if kind == "reference_call" else y

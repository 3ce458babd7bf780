"""Performance cases: the transforms users of this library run.

A case is one plan (or a batch of plans) and one pass over it:

  kind "exec"    execute() of a plan whose points are set: every iteration of
                 a solver on a fixed trajectory;
  kind "points"  set_pts() and execute(): the points move between calls
                 (motion correction, adaptive sampling, particle data);
  kind "batch"   cufinufft_batch.execute() over many plans of uneven size.

Fields: type (1: nonuniform to modes, 2: modes to nonuniform), dim, n0/n1/n2
(C-ordered modes, the last one fastest), m (points), dist (how the points
lie), f64, eps, ntr (transforms per execute), maxbatch, method (-1: the
options' default, else gpu_method), horner (gpu_kerevalmeth), tolrule (the
tolerance-meeting kernel width).
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda"


def _case(name, kind, type_, modes, m, dist, f64, eps, ntr=1, maxbatch=1, method=-1, horner=0, tolrule=0, plans=1):
    n = list(modes) + [1, 1]
    c = {"name": name, "kind": kind, "type": type_, "dim": len(modes), "n0": n[0], "n1": n[1], "n2": n[2], "m": m,
         "dist": dist, "f64": bool(f64), "eps": eps, "ntr": ntr, "maxbatch": maxbatch, "method": method,
         "horner": horner, "tolrule": tolrule, "plans": plans}
    if name is None:
        del c["name"]
    return c


def listed():
    return [
        # the smallest call: a short irregular time series evaluated from its
        # spectrum in double precision; launches and latency are all there is
        _case("series-1d-t2-f64", "exec", 2, (1001,), 2003, "series", True, 1e-9),
        # a gridding step whose points move every call (256^2 image, 1e5
        # points, the library's default options): sort, spread, FFT
        _case("moving-2d-t1-f32", "points", 1, (256, 256), 100000, "uniform", False, 1e-5),
        # radial MRI, forward operator of an iterative reconstruction (512
        # spokes x 2048 samples), layout chosen by the library
        _case("radial-2d-t2-f32", "exec", 2, (1024, 1024), 1 << 20, "radial", False, 1e-6, method=0, tolrule=1),
        # multi-coil MRI: 12 coils on one radial trajectory, odd image size,
        # default options, the default batch size of the C interface
        _case("coils-2d-t2-f32", "exec", 2, (320, 321), 201 * 1003, "radial", False, 1e-5, ntr=12, maxbatch=0),
        # the radial forward operator in double precision near full accuracy
        _case("radial-2d-t2-f64", "exec", 2, (1024, 1024), 1 << 20, "radial", True, 1e-12, method=0, horner=1,
              tolrule=1),
        # large 3D spread of half-clustered particles (cosmology, MD, cryo-EM)
        _case("cluster-3d-t1-f32", "exec", 1, (128, 128, 128), 32000000, "cluster", False, 1e-6, method=0, tolrule=1),
        # fields at the same particles in double precision: the largest case
        _case("cluster-3d-t2-f64", "exec", 2, (128, 128, 128), 32000000, "cluster", True, 1e-9, method=0, horner=1,
              tolrule=1),
        # double-precision 3D adjoint, odd and uneven image, default options
        _case("volume-3d-t1-f64", "exec", 1, (81, 96, 75), 2000000, "uniform", True, 1e-9),
        # long irregular time series to its spectrum, default options
        _case("series-1d-t1-f32", "exec", 1, (1000000,), 10000000, "series", False, 1e-6),
        # a volume evaluated at points that move every call, default options
        _case("moving-3d-t2-f32", "points", 2, (100, 81, 64), 1000003, "uniform", False, 1e-5),
        # spectrum to many irregular times in double precision, default options
        _case("long-1d-t2-f64", "exec", 2, (200001,), 3000000, "uniform", True, 1e-11),
        # many uneven 2D gridding problems executed together
        _case("batch-2d-t1-f32", "batch", 1, (256, 256), 150000, "uniform", False, 1e-5, method=0, tolrule=1,
              plans=64),
    ]


# ---------------------------------------------------------------------------
def _width(eps, f64):
    return min(16, max(2, math.ceil(-math.log10(max(eps, 1e-15 if f64 else 1e-7) / 10.0))))


def _modes(c):
    return tuple(c["n%d" % d] for d in range(c["dim"]))


def _batch_specs(c):
    """Sizes of a batch's plans: modes from a quarter to four times the named
    size (per axis half to twice), points likewise, one stream of numbers."""
    r = np.random.RandomState(1234 + c["plans"])
    specs = []
    for _ in range(c["plans"]):
        modes = tuple(max(8, int(n * 2.0 ** r.uniform(-1, 1))) for n in _modes(c))
        specs.append((modes, max(16, int(c["m"] * 4.0 ** r.uniform(-1, 1)))))
    return specs


def _cost(c):
    """Weighted kernel taps, plus the grid."""
    ns = _width(c["eps"], c["f64"]) + c["tolrule"]
    slow = c["f64"] and c["eps"] < 1e-6
    total = 0.0
    for modes, m in (_batch_specs(c) if c["kind"] == "batch" else [(_modes(c), c["m"])]):
        grid = float(np.prod([2.0 * n for n in modes]))
        total += c["ntr"] * (m * float(ns) ** len(modes) * (6 if slow else 1) + 20 * grid * (4 if slow else 1))
    return total


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges."""
    most = 6 * 32e6 * 11.0 ** 3
    while True:
        kind = rng.choice(["exec"] * 5 + ["points"] * 3 + ["batch"])
        dim = rng.choice([1, 2, 2, 3])
        f64 = rng.random() < 0.45
        eps = rng.choice([1e-6, 1e-9, 1e-11, 1e-12] if f64 else [1e-3, 1e-4, 1e-5, 1e-6])
        type_ = rng.choice([1, 2])
        if kind == "batch":
            dim, f64, eps = 2, False, rng.choice([1e-4, 1e-5])
        if dim == 1:
            modes = (_log(rng, 1000, 1000000),)
            m = _log(rng, 2000, 10000000)
            dist = rng.choice(["uniform", "series"])
        elif dim == 2:
            n = _log(rng, 100, 1024)
            modes = (n, max(64, int(n * rng.uniform(0.7, 1.0))))
            m = _log(rng, 20000, 4000000)
            dist = rng.choice(["uniform", "radial", "cluster"])
        else:
            n = _log(rng, 32, 128)
            modes = (n, max(24, int(n * rng.uniform(0.7, 1.0))), max(24, int(n * rng.uniform(0.7, 1.0))))
            m = _log(rng, 100000, 32000000 if not f64 else 4000000)
            dist = rng.choice(["uniform", "cluster"])
        ntr, maxbatch = 1, 1
        if kind == "exec" and dim < 3 and rng.random() < 0.3:
            ntr, maxbatch = rng.randint(2, 16), rng.choice([0, 0, 1, 4])
        method = rng.choice([-1, -1, 0])
        plans = 1
        if kind == "batch":
            plans, method = rng.randint(8, 64), 0
            modes = tuple(min(n, 400) for n in modes)
            m = min(m, 300000)
            dist = "uniform"
        c = _case(None, kind, type_, modes, m, dist, f64, eps, ntr, maxbatch, method, rng.choice([0, 0, 1]),
                  rng.choice([0, 1]), plans)
        if _cost(c) <= 0.5 * most and c["ntr"] * c["m"] * c["plans"] <= 40000000:
            return c


# ---------------------------------------------------------------------------
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _points(dim, m, dist, seed, salt):
    """Coordinates in [-pi, pi), FP64 on the device."""
    g = _gen(seed, 17 + salt)
    pi = math.pi

    def uniform(n):
        return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (2 * pi) - pi

    if dist == "series":  # ordered times with jitter
        t = torch.arange(m, device=DEV, dtype=torch.float64)
        j = torch.rand(m, generator=g, device=DEV, dtype=torch.float64)
        return [(t + j) * (2 * pi / m) - pi]
    if dist == "radial":  # golden-angle spokes through the centre, a random first angle
        samples = max(64, int(round(2.0 * math.sqrt(m))))
        samples = min(m, samples)
        k = torch.arange(m, device=DEV, dtype=torch.float64)
        spoke = torch.floor(k / samples)
        first = float(torch.rand(1, generator=g, device=DEV, dtype=torch.float64)) * pi
        th = spoke * (pi * (3.0 - math.sqrt(5.0))) + first
        r = (k - spoke * samples) * (2 * pi / samples) - pi
        return [r * torch.sin(th), r * torch.cos(th)]
    if dist == "cluster":  # half uniform, half in 8 Gaussian clusters
        h = m // 2
        centre = torch.rand(8, dim, generator=g, device=DEV, dtype=torch.float64) * (2 * pi) - pi
        which = torch.randint(0, 8, (m - h,), generator=g, device=DEV)
        out = []
        for d in range(dim):
            x = centre[which, d] + 0.05 * torch.randn(m - h, generator=g, device=DEV, dtype=torch.float64)
            out.append(torch.cat([uniform(h), torch.remainder(x + pi, 2 * pi) - pi]))
        return out
    return [uniform(m) for _ in range(dim)]


def _inputs(c, seed):
    """Per plan: modes, m, coordinates (C-ordered axes) and the input values,
    in the plan's precision."""
    rdt, cdt = (torch.float64, torch.complex128) if c["f64"] else (torch.float32, torch.complex64)
    specs = _batch_specs(c) if c["kind"] == "batch" else [(_modes(c), c["m"])]
    out = []
    for i, (modes, m) in enumerate(specs):
        pts = []
        for p in _points(len(modes), m, c["dist"], seed, 101 * i):
            q = p.to(rdt)
            pts.append(torch.where(q >= math.pi, torch.full_like(q, -math.pi), q).contiguous())
        shape = (c["ntr"], m) if c["type"] == 1 else (c["ntr"],) + modes
        g = _gen(seed, 50021 + i)
        v = torch.randn(*shape, 2, generator=g, device=DEV, dtype=rdt)
        out.append((modes, m, pts, torch.view_as_complex(v).to(cdt)))
    return out


def _plan(c, modes):
    from cufinufft_gb300 import cufinufft
    kw = {"gpu_kerevalmeth": c["horner"], "maxbatchsize": c["maxbatch"]}
    if c["method"] >= 0:
        kw["gpu_method"] = c["method"]
    if c["tolrule"]:
        kw["width_rule"] = "tol"
    return cufinufft(c["type"], modes, n_trans=c["ntr"], eps=c["eps"], dtype=np.float64 if c["f64"] else np.float32,
                     **kw)


def prepare(case, seed):
    parts = []
    for modes, m, pts, v in _inputs(case, seed):
        plan = _plan(case, modes)
        if case["kind"] != "points":
            plan.set_pts(*pts)
        out = torch.empty((case["ntr"],) + (modes if case["type"] == 1 else (m,)), dtype=v.dtype, device=DEV)
        c, fk = (v, out) if case["type"] == 1 else (out, v)
        parts.append({"plan": plan, "pts": pts, "c": c, "fk": fk, "out": out})
    state = {"kind": case["kind"], "parts": parts}
    if case["kind"] == "batch":
        from cufinufft_gb300 import cufinufft_batch
        state["batch"] = cufinufft_batch([p["plan"] for p in parts])
        state["c"] = [p["c"] for p in parts]
        state["fk"] = [p["fk"] for p in parts]
    return state


def run(state):
    if state["kind"] == "batch":
        state["batch"].execute(state["c"], state["fk"])
        return [p["out"] for p in state["parts"]]
    p = state["parts"][0]
    if state["kind"] == "points":
        p["plan"].set_pts(*p["pts"])
    p["plan"].execute(p["c"], p["fk"])
    return p["out"]


def work(case):
    """Coordinates and values read once, results written once; the kernel's
    multiply-adds and a complex FFT of the twofold grid."""
    s = 8 if case["f64"] else 4
    ns = _width(case["eps"], case["f64"]) + case["tolrule"]
    nbytes = flops = 0.0
    for modes, m in (_batch_specs(case) if case["kind"] == "batch" else [(_modes(case), case["m"])]):
        n = float(np.prod([float(k) for k in modes]))
        grid = float(np.prod([2.0 * k for k in modes]))
        nbytes += m * len(modes) * s + case["ntr"] * 2.0 * s * (m + n)
        flops += case["ntr"] * (4.0 * m * float(ns) ** len(modes) + 5.0 * grid * math.log2(grid))
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# The sums in FP64 without a kernel: exp(i k x) about the nearest point g h of
# a grid at least twice as fine as the modes,
#   exp(i k x) = exp(i k g h) sum_p (i k (x - g h))^p / p!,
# whose terms fall below 1e-16 within a few dozen (|k (x - g h)| <= pi / 4), so
# a transform is a sum of plain FFTs of scattered (type 1) or gathered (type
# 2) moments.
_TERM = 2e-16
_MOST_TERMS_POINTS = 4.0e9


def _terms(modes, sizes):
    a = [(n / 2.0) * math.pi / size for n, size in zip(modes, sizes)]
    bound = [[x ** p / math.factorial(p) for p in range(40)] for x in a]
    terms = [((), 1.0)]
    for b in bound:
        terms = [(t + (p,), w * b[p]) for t, w in terms for p in range(40) if w * b[p] > _TERM]
    return [t for t, _ in terms]


def _grid_sizes(modes):
    out = []
    for n in modes:
        size = 2 * n if len(modes) > 1 else 4 * n
        while True:  # a size the FFT likes
            k = size
            for q in (2, 3, 5):
                while k % q == 0:
                    k //= q
            if k == 1:
                break
            size += 1
        out.append(size)
    return out


def _exact_one(type_, modes, pts, values, sign):
    dim = len(modes)
    sizes = _grid_sizes(modes)
    cells = int(np.prod(sizes))
    m = pts[0].numel()
    idx = torch.zeros(m, dtype=torch.int64, device=DEV)
    off = []
    for p, size in zip(pts, sizes):
        x = p.double()
        h = 2 * math.pi / size
        g = torch.round(x / h)
        off.append((x - g * h) / (h / 2))  # in [-1, 1]
        idx = idx * size + torch.remainder(g.long(), size)
    ks = [torch.arange(n, device=DEV, dtype=torch.float64) - n // 2 for n in modes]
    slot = [torch.remainder(torch.arange(n, device=DEV) - n // 2, size) for n, size in zip(modes, sizes)]

    def axis(v, d):
        return v.reshape([-1 if e == d else 1 for e in range(dim)])

    def weight(t):
        w = torch.ones([1] * dim, dtype=torch.complex128, device=DEV)
        for d, p in enumerate(t):
            h = 2 * math.pi / sizes[d]
            w = w * axis(((1j * sign * h / 2) * ks[d]) ** p / math.factorial(p), d)
        return w

    def corner(full):
        for d in range(dim):
            full = full.index_select(d, slot[d])
        return full

    def power(t):
        w = torch.ones(m, dtype=torch.float64, device=DEV)
        for d, p in enumerate(t):
            if p:
                w = w * off[d] ** p
        return w

    outs = []
    for v in values.to(torch.complex128):
        total = torch.zeros(modes if type_ == 1 else (m,), dtype=torch.complex128, device=DEV)
        for t in _terms(modes, sizes):
            if type_ == 1:
                mom = torch.zeros(cells, 2, dtype=torch.float64, device=DEV)
                mom.index_add_(0, idx, torch.view_as_real(v * power(t)))
                f = torch.view_as_complex(mom).reshape(sizes)
                f = torch.fft.ifftn(f, norm="forward") if sign > 0 else torch.fft.fftn(f)
                total += corner(f) * weight(t)
            else:
                full = torch.zeros(sizes, dtype=torch.complex128, device=DEV)
                at = torch.zeros([1] * dim, dtype=torch.int64, device=DEV)
                for d in range(dim):
                    at = at * sizes[d] + axis(slot[d], d)
                full.view(-1)[at.reshape(-1)] = (v * weight(t)).reshape(-1)
                f = torch.fft.ifftn(full, norm="forward") if sign > 0 else torch.fft.fftn(full)
                total += f.reshape(-1)[idx] * power(t)
        outs.append(total)
    return torch.stack(outs)


def exact(case, seed):
    terms = 0.0
    for modes, m in (_batch_specs(case) if case["kind"] == "batch" else [(_modes(case), case["m"])]):
        sizes = _grid_sizes(modes)
        terms += case["ntr"] * len(_terms(modes, sizes)) * (m + 0.5 * float(np.prod(sizes)))
    if terms > _MOST_TERMS_POINTS * 3:
        return None
    sign = 1 if case["type"] == 1 else -1
    got = [_exact_one(case["type"], modes, pts, v, sign) for modes, m, pts, v in _inputs(case, seed)]
    return got if case["kind"] == "batch" else got[0]

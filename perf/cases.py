"""Workloads of the density estimators, as a program of their users runs them.

Each case is one estimation (or one batch call) through the public API: the samples and the
grid are at hand, the call returns the density on the grid and the selected bandwidth step of
every grid point.  The grids are those of the reference's own benchmark and tests (100 to 2500
points in 1-D, 33^2 to 300^2 in 2-D, 150 points an axis by default), of this repository's
benchmark (1,024 points, 512^2, 128^3, the batched mixes), and odd ones.

entry   "api":    initialize_estimation / estimate_density / get_density on host samples
        "device": raw.gradepro_device, samples and results stay on the GPU
        "batch":  raw.gradepro_batch, several estimations of mixed shapes in one call
        "rot":    raw.rot, the rule-of-thumb estimator, on the GPU
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "parallelkde.jl_b200"))
import pkde_b200 as pk  # noqa: E402
from pkde_b200 import raw  # noqa: E402


def _case(name, entry, dims, n, boots, steps, dist, pad=0.1):
    d = list(dims) + [0] * (4 - len(dims))
    c = {"entry": entry, "d1": d[0], "d2": d[1], "d3": d[2], "d4": d[3], "n": n, "boots": boots, "steps": steps,
         "dist": dist, "pad": pad}
    return dict(c, name=name) if name else c


def _batch(name, count, mix):
    c = {"entry": "batch", "count": count, "mix": mix, "boots": 32, "steps": 100}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's benchmark and its end-to-end test: N(0, 1) on [-8, 8], default bootstraps
        # and steps; the smallest calls, where launches and host work count
        _case("1d_500_api", "api", (500,), 1000, 100, 250, "normal"),
        # 1-D of the repository's benchmark: a power of two, the range padded by 3 standard deviations
        _case("1d_1024", "device", (1024,), 10_000, 100, 250, "normal", 3.0),
        # the longest 1-D grid of the reference's benchmark
        _case("1d_2500", "device", (2500,), 100_000, 100, 250, "normal"),
        # the reference's 2-D benchmark through the host API
        _case("2d_100_api", "api", (100, 100), 100_000, 100, 250, "normal"),
        # the default grid (150 points an axis) with unequal odd sizes beside it
        _case("2d_150x77", "device", (150, 77), 10_000, 100, 250, "mixture"),
        # the default workload of bench.py
        _case("2d_512", "device", (512, 512), 1_000_000, 64, 200, "mixture"),
        # the most frequent kind of the batched mix, a mixed-radix cube
        _case("3d_96", "device", (96, 96, 96), 200_000, 32, 100, "mixture"),
        # a small cube with odd sizes
        _case("3d_50x41x36", "device", (50, 41, 36), 20_000, 32, 100, "mixture"),
        # the largest workload of the benchmark
        _case("3d_128", "device", (128, 128, 128), 4_000_000, 32, 150, "banana"),
        # the smaller 4-D requests of the served mix
        _case("4d_24", "device", (24, 24, 24, 24), 100_000, 32, 100, "mixture"),
        # many small estimations in one call
        _batch("batch_small_24", 24, 11),
        # one rule-of-thumb density of a large sample
        _case("rot_2d_300", "rot", (300, 300), 1_000_000, 0, 0, "mixture"),
    ]


def _primes(n):
    out, p = [], 2
    while n > 1:
        while n % p == 0:
            out.append(p)
            n //= p
        p += 1
    return out


def _axis(r, lo, hi):
    """An axis length: mostly round numbers and powers of two, a quarter of them anything."""
    v = math.exp(r.uniform(math.log(lo), math.log(hi)))
    kind = r.random()
    if kind < 0.45:
        v = 10 * round(v / 10)
    elif kind < 0.75:
        v = r.choice([2 ** k for k in range(4, 13)] + [3 * 2 ** k for k in range(4, 8)] + [5 * 2 ** k for k in range(3, 7)])
    return min(hi, max(lo, int(round(v))))


def draw(rng):
    while True:
        kind = rng.choice(["1d", "1d", "2d", "2d", "2d", "3d", "4d", "batch", "rot"])
        if kind == "batch":
            return _batch(None, rng.randint(8, 32), rng.randint(12, 10 ** 6))
        ndim = rng.randint(1, 3) if kind == "rot" else int(kind[0])
        lo, hi = {1: (100, 4096), 2: (33, 512), 3: (32, 128), 4: (16, 32)}[ndim]
        dims = [_axis(rng, lo, hi) for _ in range(ndim)]
        if rng.random() < 0.5:  # equal axes are the common request
            dims = [dims[0]] * ndim
        n = int(round(math.exp(rng.uniform(math.log(1e3), math.log(2e6)))))
        boots, steps = rng.choice([32, 64, 100]), rng.choice([100, 150, 200, 250])
        if kind == "rot":
            return _case(None, "rot", dims, n, 0, 0, "mixture")
        # a cost below the largest listed case's; an axis costs about the sum of its radices
        g = math.prod(dims)
        cost = (steps + 1) * (boots + 1) * g * sum(5 + sum(p for p in _primes(d) if p > 5) for d in dims)
        if cost <= 6e10 and n * (boots + 1) <= 1e8:
            return _case(None, rng.choice(["api", "device"]), dims, n, boots, steps, rng.choice(["normal", "mixture"]))


def work(case):
    """Samples in, density and selected steps out; the inverse transforms of every bandwidth step
    (two real arrays a complex transform) and the variance update of each bootstrap."""
    if case["entry"] == "batch":
        w = [work(c) for c in _members(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    dims = _dims(case)
    g = math.prod(dims)
    if case["entry"] == "rot":
        return {"bytes": 8 * len(dims) * case["n"] + 8 * g, "flops": 2 * 2.5 * g * math.log2(g)}
    arrays = 2 * ((case["boots"] + 1) // 2) + 1
    s = case["steps"] + 1
    return {"bytes": 8 * len(dims) * case["n"] + 12 * g,
            "flops": s * g * (arrays * 5 * math.log2(g) + 15 * case["boots"])}


def _dims(case):
    return tuple(case[k] for k in ("d1", "d2", "d3", "d4") if case[k])


def _members(case):
    """The estimations of a batch call: 1-D grids of 256 to 1024 points and 2-D grids of 64^2 to
    128^2, sample counts log-uniform in 1e3 to 1e4; an odd size now and then."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(1e3), math.log(1e4)))))
        dims = (r.choice([256, 500, 512, 1024]),) if r.random() < 0.5 else (r.choice([64, 96, 100, 128]),) * 2
        out.append(_case(None, "device", dims, n, case["boots"], case["steps"], "mixture"))
    return out


def _samples(case, seed):
    """(n, N) float64 samples on the GPU, from the seed alone."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    N, n = len(_dims(case)), case["n"]

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    if case["dist"] == "normal":
        return normal(n, N)
    if case["dist"] == "banana":  # 70 % banana, 30 % Student-t with 3 degrees of freedom
        nt = n - int(0.7 * n)
        x = normal(n, N)
        x[:, 1] = 0.5 * x[:, 0] ** 2 + 0.3 * x[:, 1]
        x[:nt] = normal(nt, N) / (normal(nt, 3).square().sum(1, keepdim=True) / 3).sqrt()
        return x
    r = random.Random(int(seed))  # a Gaussian mixture of three components
    which = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    x, out = normal(n, N), torch.empty(n, N, device="cuda", dtype=torch.float64)
    for c, (lo, hi) in enumerate(((0.0, 0.5), (0.5, 0.8), (0.8, 2.0))):
        a = torch.tensor([[r.gauss(0, 0.3) + (r.uniform(0.6, 1.2) if i == j else 0) for j in range(N)] for i in range(N)],
                         device="cuda", dtype=torch.float64)
        mu = torch.tensor([r.uniform(-3, 3) for _ in range(N)], device="cuda", dtype=torch.float64)
        sel = (which >= lo) & (which < hi)
        out[sel] = (x @ a.T + mu)[sel]
    return out


def _ranges(case, x):
    """(low, high, points) of each axis: the benchmark's [-8, 8], or the extrema padded."""
    dims = _dims(case)
    if case["dist"] == "normal" and case["pad"] == 0.1:
        return [(-8.0, 8.0, d) for d in dims]
    lo, hi = x.min(0).values.cpu().numpy(), x.max(0).values.cpu().numpy()
    pad = case["pad"] * (x.std(0).cpu().numpy() if case["pad"] >= 1 else hi - lo)
    return [(float(a), float(b), d) for a, b, d in zip(lo - pad, hi + pad, dims)]


def _job(case, seed):
    x = _samples(case, seed).contiguous()
    grid = pk.initialize_grid(_ranges(case, x))
    g = math.prod(_dims(case))
    return {"grid": grid, "data": x, "density": torch.empty(g, dtype=torch.float64, device="cuda"),
            "selected": torch.empty(g, dtype=torch.int32, device="cuda"), "seed": int(seed),
            "n_bootstraps": case["boots"], "n_steps": case["steps"]}


def prepare(case, seed):
    if case["entry"] == "batch":
        return {"entry": "batch", "jobs": [_job(c, seed * 1000 + k) for k, c in enumerate(_members(case))]}
    if case["entry"] == "api":
        x = _samples(case, seed)
        grid = pk.initialize_grid(_ranges(case, x))
        est = pk.initialize_estimation(np.ascontiguousarray(x.T.cpu().numpy()), grid=grid)
        return {"entry": "api", "est": est,
                "kw": {"n_bootstraps": case["boots"], "n_steps": case["steps"], "seed": int(seed)}}
    return dict(_job(case, seed), entry=case["entry"])


def run(state):
    if state["entry"] == "batch":
        raw.gradepro_batch(state["jobs"], device=True)
        return [{"density": j["density"], "selected": j["selected"]} for j in state["jobs"]]
    if state["entry"] == "api":
        pk.estimate_density(state["est"], "gradepro", **state["kw"])
        return {"density": pk.get_density(state["est"]), "selected": state["est"].selected_step}
    if state["entry"] == "rot":
        return {"density": raw.rot(state["grid"], state["data"], density=state["density"], device=True)}
    raw.gradepro_device(state["grid"], state["data"], state["data"].shape[0], state["density"], state["selected"],
                        seed=state["seed"], n_bootstraps=state["n_bootstraps"], n_steps=state["n_steps"])
    return {"density": state["density"], "selected": state["selected"]}


# ---------------------------------------------------------------- the same in plain torch
def exact(case, seed):
    """The densities in 64 bits (the selected steps have no value of their own: where a decision
    lies within rounding of its threshold, each implementation decides it for itself)."""
    if case["entry"] == "batch":
        return [{"density": _plain(c, seed * 1000 + k), "selected": None} for k, c in enumerate(_members(case))]
    if case["entry"] == "rot":
        return {"density": _plain(case, seed)}
    d = _plain(case, seed)
    return {"density": d.reshape(tuple(reversed(_dims(case)))) if case["entry"] == "api" else d, "selected": None}


def _mix64(x):
    def shr(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)

    def c(v):
        return v - (1 << 64) if v >> 63 else v

    x = (x ^ shr(x, 30)) * c(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * c(0x94D049BB133111EB)
    return x ^ shr(x, 31)


def _plain(case, seed):
    """Cloud-in-cell binning, spectra, and for :gradepro the bandwidth ladder with its rule."""
    x = _samples(case, seed)
    dims, n, N = _dims(case), case["n"], len(_dims(case))
    g = math.prod(dims)
    lo, hi, _ = zip(*_ranges(case, x))
    lo, hi = (torch.tensor(v, device="cuda", dtype=torch.float64) for v in (lo, hi))
    h = (hi - lo) / (torch.tensor(dims, device="cuda", dtype=torch.float64) - 1)
    cell = ((x - lo) / h).floor()
    rh = torch.fmod(x - lo, h)
    cell = cell.long()
    stride = [math.prod(dims[:j]) for j in range(N)]
    vol = float(h.prod())
    corners = []
    for c in range(1 << N):
        at, w = torch.zeros_like(cell[:, 0]), torch.full_like(rh[:, 0], 1.0 / (n * vol * vol))
        for j in range(N):
            up = (c >> j) & 1
            at = at + (cell[:, j] + up) * stride[j]
            w = w * (rh[:, j] if up else h[j] - rh[:, j])
        corners.append((at, w))
    shape = tuple(reversed(dims))

    def bin(weight, square):
        out = torch.zeros(g, device="cuda", dtype=torch.float64)
        for at, w in corners:
            v = w * w if square else w
            out.index_add_(0, at, v if weight is None else v * weight)
        return torch.fft.rfftn(out.reshape(shape))

    k = [2 * math.pi * torch.fft.fftfreq(d, float(h[j]), device="cuda", dtype=torch.float64) for j, d in enumerate(dims)]
    k[0] = k[0][:dims[0] // 2 + 1].abs()

    def gauss(t):
        p = torch.ones((), device="cuda", dtype=torch.float64)
        for j in range(N):
            p = p * torch.exp(-0.5 * (k[j] * t[j]) ** 2).reshape([-1 if N - 1 - a == j else 1 for a in range(N)])
        return p

    axes = tuple(range(-N, 0))
    full = bin(None, False)
    std = x.std(0).tolist()
    t0 = [float(v) / 2 for v in h]
    if case["entry"] == "rot":
        t = [n ** (-1.0 / (N + 4)) * s - a for s, a in zip(std, t0)]
        return torch.fft.irfftn(full * gauss(t), s=shape, dim=axes).abs().reshape(-1)
    B, S = case["boots"], case["steps"]
    m, v = [], []
    for b in range(B):
        gamma = torch.arange(b * n + 1, b * n + n + 1, device="cuda") * (0x9E3779B97F4A7C15 - (1 << 64)) + int(seed)
        pick = (((_mix64(gamma) >> 32) & 0xFFFFFFFF) * n) >> 32
        times = torch.bincount(pick, minlength=n).double()
        m.append(bin(times, False))
        v.append(bin(times, True))
    m, v = torch.stack(m), torch.stack(v)
    final = [(4 / ((N + 2) * n)) ** (1 / (N + 4)) * s for s in std]
    low_limit, over_limit = round((0.0 if N == 1 else 0.06) * S), round(0.1 * S)
    eps = 2.0 if N == 1 else -0.5
    nan = torch.full(shape, math.nan, device="cuda", dtype=torch.float64)
    density, least, f1, f2 = nan.clone(), nan.clone(), nan, nan
    low, over = torch.zeros(shape, device="cuda"), torch.zeros(shape, device="cuda")
    flag = torch.zeros(shape, device="cuda", dtype=torch.bool)
    before = math.prod(a * a for a in t0)
    for s in range(S + 1):
        t = [f / S * s for f in final]
        det = math.prod(a * a + b * b for a, b in zip(t, t0))
        dlogt, before = math.log(det / before), det
        p = gauss(t)
        mean = torch.fft.irfftn(full * p, s=shape, dim=axes).abs()
        count, avg, m2 = 0, torch.zeros_like(mean), torch.zeros_like(mean)
        step = max(1, (1 << 27) // g)
        for b in range(0, B, step):
            a = torch.fft.irfftn(m[b:b + step] * p, s=shape, dim=axes).abs() / n
            c = torch.fft.irfftn(v[b:b + step] * (p.sqrt() * (math.prod(t0) / math.sqrt(det))), s=shape, dim=axes).abs() / n
            r = (c - a * a) / a
            mb, k2 = r.mean(0), r.shape[0]
            m2 = m2 + ((r - mb) ** 2).sum(0) + (mb - avg) ** 2 * (count * k2 / (count + k2))
            avg = avg + (mb - avg) * (k2 / (count + k2))
            count += k2
        f = m2 / (B - 1) * (det ** 1.5 * float(n) ** 3)
        f = torch.where(f.isfinite(), f.log(), nan)
        d1 = ((f - f1) / (2 * dlogt if dlogt else math.nan)).abs().log()
        d2 = ((f - 2 * f1 + f2) / (dlogt * dlogt if dlogt else math.nan)).abs().log()
        below, unset = d2 < eps, least.isnan()
        first = ~flag & below & ((d1 < least) | unset) & (over <= over_limit)
        late = flag & below & unset
        over = torch.where(first, torch.zeros_like(over), over + (~flag & below & ~first).float())
        low = low + (~flag & ~below).float()
        flip = ~flag & ~below & (low > low_limit)
        least = torch.where(first | late, d1, least)
        least = torch.where(flip, nan, least)
        density = torch.where(first | late, mean, density)
        flag = flag | flip
        f1, f2 = f, f1
    return torch.where(density.isnan(), mean, density).reshape(-1)

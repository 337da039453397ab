"""Performance cases: the transforms that programs built on nufftax_b200 run.

A case is one unit of work as a program does it, through the public entry points
with inputs on the device: a type-1 / type-2 pair on points that are new in each
pass, the normal operator of an iterative reconstruction on fixed points, a
gradient step, a type 3, or a batched plan.  `listed()` names the ordinary ones,
`draw(rng)` gives more of the same ranges, `prepare` makes a program's inputs,
`run` is one pass, `work` counts what a pass cannot do without, and `exact`
evaluates the same sums directly in 64 bits.

Coordinates follow the distributions transforms meet: uniform in [-pi, pi),
clustered N(0, 0.3^2) per axis, or radial spokes (2D: golden angles; samples
uniform along the spoke).  Strengths and modes are complex standard normal.
"""

from __future__ import annotations

import math
import random

import torch

import nufftax_b200 as nb
from nufftax_b200.batch import BatchPlan

PI = math.pi
TYPE1 = {1: nb.nufft1d1, 2: nb.nufft2d1, 3: nb.nufft3d1}
TYPE2 = {1: nb.nufft1d2, 2: nb.nufft2d2, 3: nb.nufft3d2}


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _pair(dim, M, n, eps, points, c128=False, **more):
    return {"kind": "pair", "dim": dim, "M": M, "n1": n[0], "n2": n[1] if dim > 1 else 1, "n3": n[2] if dim > 2 else 1,
            "eps": eps, "points": points, "c128": c128, **more}


def listed():
    return [
        # one small request, a served stream's smallest: latency and launches
        _pair(2, 1000, (128, 128), 1e-6, "uniform", name="2d_small"),
        # the plain 1D workload: type 1 then type 2 of 200,000 points
        _pair(1, 200_000, (8192,), 1e-6, "uniform", name="1d_plain"),
        # MR imaging, radial trajectory of 512 spokes x 1024 samples, gridding and
        # degridding once each
        _pair(2, 524_288, (512, 512), 1e-6, "radial", name="2d_radial"),
        # many points packed into a few pixels: 4 million, Gaussian-clustered
        _pair(2, 4_000_000, (512, 512), 1e-6, "clustered", name="2d_clustered"),
        # low accuracy on ragged sizes (previews, learned reconstructions)
        _pair(2, 300_007, (243, 181), 1e-3, "uniform", name="2d_low_accuracy"),
        # scientific double precision at its tightest tolerance
        _pair(2, 200_003, (255, 192), 1e-12, "uniform", c128=True, name="2d_double"),
        # a 3D request of ordinary size
        _pair(3, 1_000_000, (96, 112, 128), 1e-6, "uniform", name="3d_request"),
        # one iteration of a multi-coil reconstruction: fixed trajectory, the normal
        # operator (type 2, then its adjoint) over 8 coils in one call each
        {"kind": "normal", "dim": 2, "M": 262_144, "n1": 256, "n2": 256, "n3": 1, "eps": 1e-6, "points": "radial",
         "c128": False, "coils": 8, "name": "2d_coils"},
        # differentiated 3D type 1: gradients of a least-squares loss with respect to
        # the strengths and all coordinates, 8 million points
        {"kind": "grad1", "dim": 3, "M": 8_000_000, "n1": 128, "n2": 128, "n3": 128, "eps": 1e-6, "points": "uniform",
         "c128": False, "name": "3d_gradient"},
        # trajectory learning: type 2 with gradients of the image and the coordinates
        {"kind": "grad2", "dim": 2, "M": 262_144, "n1": 256, "n2": 256, "n3": 1, "eps": 1e-6, "points": "radial",
         "c128": False, "name": "2d_trajectory_gradient"},
        # 2D type 3 between scattered points, targets in [-300, 300]^2
        {"kind": "type3", "M": 100_000, "K": 100_000, "extent": 300.0, "eps": 1e-6, "name": "2d_type3"},
        # many uneven 2D problems in one plan, type 1 and type 2 of each
        {"kind": "batched", "problems": 24, "sizes": 77, "M_low": 10_000, "M_high": 2_000_000, "eps": 1e-5,
         "name": "2d_batched"},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the listed ranges (sizes log-uniform, odd ones among them)."""
    kind = rng.choice(["pair1", "pair2", "pair2", "pair2", "pair3", "pair3", "double", "normal", "grad1", "grad2",
                       "type3", "batched"])
    eps = rng.choice([1e-3, 1e-4, 1e-5, 1e-6, 1e-6])
    if kind == "pair1":
        return _pair(1, _log_int(rng, 1000, 2_000_000), (_log_int(rng, 200, 100_000),), eps,
                     rng.choice(["uniform", "clustered"]))
    if kind == "pair2":
        return _pair(2, _log_int(rng, 1000, 4_000_000), [_log_int(rng, 100, 600) for _ in range(2)], eps,
                     rng.choice(["uniform", "clustered", "radial"]))
    if kind == "pair3":
        return _pair(3, _log_int(rng, 10_000, 4_000_000), [_log_int(rng, 40, 140) for _ in range(3)], eps,
                     rng.choice(["uniform", "uniform", "clustered"]))
    if kind == "double":
        dim = rng.choice([1, 2, 2, 3])
        n = {1: (200, 50_000), 2: (64, 400), 3: (24, 64)}[dim]
        return _pair(dim, _log_int(rng, 1000, 100_000 if dim == 3 else 500_000), [_log_int(rng, *n) for _ in range(dim)],
                     rng.choice([1e-6, 1e-9, 1e-12] if dim < 3 else [1e-6, 1e-9]), rng.choice(["uniform", "clustered"]),
                     c128=True)
    if kind == "normal":
        return {"kind": "normal", "dim": 2, "M": _log_int(rng, 20_000, 500_000), "n1": _log_int(rng, 128, 384),
                "n2": _log_int(rng, 128, 384), "n3": 1, "eps": eps, "points": rng.choice(["radial", "uniform"]),
                "c128": False, "coils": rng.choice([1, 4, 8, 12])}
    if kind in ("grad1", "grad2"):
        dim = rng.choice([2, 3])
        n = (100, 400) if dim == 2 else (40, 128)
        return {"kind": kind, "dim": dim, "M": _log_int(rng, 20_000, 2_000_000), "n1": _log_int(rng, *n),
                "n2": _log_int(rng, *n), "n3": _log_int(rng, *n) if dim == 3 else 1, "eps": eps,
                "points": rng.choice(["uniform", "radial"] if dim == 2 else ["uniform", "clustered"]), "c128": False}
    if kind == "type3":
        return {"kind": "type3", "M": _log_int(rng, 1000, 500_000), "K": _log_int(rng, 1000, 500_000),
                "extent": float(round(rng.uniform(50.0, 300.0), 1)), "eps": eps}
    return {"kind": "batched", "problems": rng.randint(4, 24), "sizes": rng.randint(0, 10_000), "M_low": 10_000,
            "M_high": 1_000_000, "eps": rng.choice([1e-4, 1e-5, 1e-6])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _points(gen, dim, M, points, dtype):
    dev = gen.device
    if points == "radial":
        spokes = max(1, M // 1024)
        s = torch.arange(M, device=dev) % spokes
        theta = (s.double() * (PI * (math.sqrt(5.0) - 1.0) / 2.0)) % PI
        r = (torch.rand(M, generator=gen, device=dev, dtype=torch.float64) * 2 - 1) * PI
        return [(r * torch.cos(theta)).to(dtype).contiguous(), (r * torch.sin(theta)).to(dtype).contiguous()][:dim]
    if points == "clustered":
        xs = [torch.randn(M, generator=gen, device=dev, dtype=torch.float64) * 0.3 for _ in range(dim)]
        return [(((x + PI) % (2 * PI)) - PI).to(dtype) for x in xs]
    return [((torch.rand(M, generator=gen, device=dev, dtype=torch.float64) * 2 - 1) * PI).to(dtype)
            for _ in range(dim)]


def _normal(gen, shape, cdtype):
    return torch.randn(shape, generator=gen, device=gen.device, dtype=cdtype)


def _n_modes(case):
    return tuple(case["n%d" % (d + 1)] for d in range(case["dim"]))


def _problems(case):
    """Sizes of a batched plan's problems: M log-uniform, modes per axis from
    {128, 256, 384, 512}, even problems uniform, odd ones clustered."""
    rng = random.Random(case["sizes"])
    out = []
    for p in range(case["problems"]):
        M = _log_int(rng, case["M_low"], case["M_high"])
        n = (rng.choice([128, 256, 384, 512]), rng.choice([128, 256, 384, 512]))
        out.append((M, n, "clustered" if p % 2 else "uniform"))
    return out


def _inputs(case, seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "batched":
        pts, c, f = [], [], []
        for M, n, points in _problems(case):
            pts.append(_points(gen, 2, M, points, torch.float32))
            c.append(_normal(gen, (M,), torch.complex64))
            f.append(_normal(gen, (n[1], n[0]), torch.complex64))
        return {"x": pts, "c": c, "f": f}
    if kind == "type3":
        x = _points(gen, 2, case["M"], "uniform", torch.float32)
        t = [((torch.rand(case["K"], generator=gen, device=gen.device) * 2 - 1) * case["extent"]) for _ in range(2)]
        return {"x": x, "t": t, "c": _normal(gen, (case["M"],), torch.complex64)}
    rdt, cdt = (torch.float64, torch.complex128) if case["c128"] else (torch.float32, torch.complex64)
    n = _n_modes(case)
    lead = (case["coils"],) if kind == "normal" else ()
    s = {"x": _points(gen, case["dim"], case["M"], case["points"], rdt)}
    if kind != "normal":
        s["c"] = _normal(gen, (case["M"],), cdt)
    s["f"] = _normal(gen, lead + tuple(reversed(n)), cdt)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "batched":
        s["plan"] = BatchPlan(s["x"], [n for _, n, _ in _problems(case)], eps=case["eps"])
    elif case["kind"] == "type3":
        e = case["extent"]
        s["grid"] = nb.compute_type3_grid_sizes_2d(PI, PI, e, e, eps=case["eps"])
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind, eps = case["kind"], case["eps"]
    if kind == "batched":
        return s["plan"].run(s["c"], s["f"])
    if kind == "type3":
        return nb.nufft2d3(*s["x"], s["c"], *s["t"], s["grid"], eps=eps)
    dim, n = case["dim"], _n_modes(case)
    if kind == "pair":
        nb.sort_cache.clear()  # the points are new: no sort of an earlier pass serves this one
        return TYPE1[dim](*s["x"], s["c"], n if dim > 1 else n[0], eps=eps), TYPE2[dim](*s["x"], s["f"], eps=eps)
    if kind == "normal":
        c = TYPE2[dim](*s["x"], s["f"], eps=eps)
        return c, TYPE1[dim](*s["x"], c, n, eps=eps)
    # a gradient step: the parameters are this step's leaves
    xs = [x.detach().requires_grad_() for x in s["x"]]
    if kind == "grad1":
        c = s["c"].detach().requires_grad_()
        f = TYPE1[dim](*xs, c, n, eps=eps)
        r = f - s["f"]
        loss = (r.real.square() + r.imag.square()).sum()
        loss.backward()
        return (f.detach(), c.grad, *[x.grad for x in xs])
    f = s["f"].detach().requires_grad_()
    c = TYPE2[dim](*xs, f, eps=eps)
    r = c - s["c"]
    loss = (r.real.square() + r.imag.square()).sum()
    loss.backward()
    return (c.detach(), f.grad, *[x.grad for x in xs])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _grid(n, eps):
    kp = nb.compute_kernel_params(eps)
    return kp.nspread, math.prod(nb.compute_grid_size(v, 2.0, kp.nspread) for v in n)


def _transform_flops(dim, M, n, eps, nt=1):
    """A type 1 or type 2: a real times a complex multiply-add per footprint cell,
    the fine grid's FFT and the deconvolution."""
    ns, cells = _grid(n, eps)
    return nt * (4.0 * M * ns ** dim + 5.0 * cells * math.log2(cells) + 2.0 * math.prod(n))


def work(case):
    kind, eps = case["kind"], case["eps"]
    if kind == "batched":
        b = fl = 0.0
        for M, n, _ in _problems(case):
            b += M * (8 + 8 + 8) + 2 * 8 * math.prod(n)
            fl += 2 * _transform_flops(2, M, n, eps)
        return {"bytes": b, "flops": fl}
    if kind == "type3":
        M, K, e = case["M"], case["K"], case["extent"]
        grid = nb.compute_type3_grid_sizes_2d(PI, PI, e, e, eps=eps)
        ns, inner = _grid(grid, eps)
        return {"bytes": M * 16.0 + K * 16.0, "flops": 4.0 * (M + K) * ns ** 2 + 5.0 * inner * math.log2(inner)}
    dim, M, n = case["dim"], case["M"], _n_modes(case)
    rb = 8 if case["c128"] else 4
    N = math.prod(n)
    t = _transform_flops(dim, M, n, eps, case.get("coils", 1))
    if kind == "pair":  # coordinates, c, f in; f, c out
        return {"bytes": rb * (M * dim + 4.0 * M + 4.0 * N), "flops": 2 * t}
    if kind == "normal":  # coordinates and f in; c and f out
        return {"bytes": rb * (M * dim + case["coils"] * (2.0 * M + 4.0 * N)), "flops": 2 * t}
    # gradients: coordinates, c, f in; the transform and every gradient out; the
    # coordinate gradients need one derivative sum per axis over the footprint
    out = 2.0 * N + 2.0 * M if kind == "grad1" else 2.0 * M + 2.0 * N
    ns, _ = _grid(n, eps)
    fl = 2 * t + 4.0 * dim * M * ns ** dim
    return {"bytes": rb * (M * dim + 2.0 * M + 2.0 * N + out + M * dim), "flops": fl}


# ---------------------------------------------------------------------------
# The same sums in 64 bits
# ---------------------------------------------------------------------------
def _chunks(M, width):
    step = max(1, min(M, (1 << 26) // max(width, 1)))
    for a in range(0, M, step):
        yield a, min(M, a + step)


def _waves(xs, n, sign, a, b):
    """e^{i sign k x_j} per axis for points a..b: (points, n_d) each."""
    out = []
    for x, nd in zip(xs, n):
        k = torch.arange(-(nd // 2), (nd + 1) // 2, device=x.device, dtype=torch.float64)
        out.append(torch.polar(torch.ones((), device=x.device, dtype=torch.float64), sign * x[a:b, None].double() * k))
    return out


def _outer(waves):
    """(points, n_d * .. * n_2) products of every axis but the first."""
    w = waves[-1]
    for e in reversed(waves[1:-1]):
        w = (w[:, :, None] * e[:, None, :]).reshape(w.shape[0], -1)
    return w


def _direct1(xs, c, n, sign):
    M = c.shape[-1]
    rest = math.prod(n[1:])
    f = torch.zeros((c.shape[0], rest, n[0]), dtype=torch.complex128, device=c.device)
    for a, b in _chunks(M, rest + sum(n)):
        w = _waves(xs, n, sign, a, b)
        o = _outer(w) if len(n) > 1 else None
        for t in range(c.shape[0]):
            ct = c[t, a:b].to(torch.complex128)
            f[t] += (w[0].T @ ct)[None, :] if o is None else (o * ct[:, None]).T @ w[0]
    return f.reshape((c.shape[0],) + tuple(reversed(n)))


def _direct2(xs, f, n, sign, grad=False):
    """Values at the points and, with `grad`, the sums with a factor i sign k_d per axis."""
    M, nt, rest = xs[0].shape[0], f.shape[0], math.prod(n[1:])
    dev = f.device
    outs = [torch.empty((nt, M), dtype=torch.complex128, device=dev) for _ in range(1 + (len(n) if grad else 0))]
    F = f.to(torch.complex128).reshape(nt, rest, n[0])
    ks = [torch.arange(-(nd // 2), (nd + 1) // 2, device=dev, dtype=torch.float64) for nd in n]
    for a, b in _chunks(M, 2 * rest + sum(n)):
        w = _waves(xs, n, sign, a, b)
        o = _outer(w) if len(n) > 1 else torch.ones((b - a, 1), dtype=torch.complex128, device=dev)
        for t in range(nt):
            h = (w[0] @ F[t].T) * o
            outs[0][t, a:b] = h.sum(1)
            if grad:
                outs[1][t, a:b] = (1j * sign) * (((w[0] * ks[0]) @ F[t].T) * o).sum(1)
                if len(n) == 2:
                    outs[2][t, a:b] = (1j * sign) * (h * ks[1]).sum(1)
                elif len(n) == 3:
                    h = h.reshape(b - a, n[2], n[1])
                    outs[2][t, a:b] = (1j * sign) * (h.sum(1) * ks[1]).sum(1)
                    outs[3][t, a:b] = (1j * sign) * (h.sum(2) * ks[2]).sum(1)
    return outs


def _too_long(case):
    """Whether the direct sums would take more than a few seconds on one GPU."""
    if case["kind"] == "batched":
        return sum(M * math.prod(n) for M, n, _ in _problems(case)) > 4e12
    if case["kind"] == "type3":
        return case["M"] * case["K"] > 3e11
    return case["M"] * math.prod(_n_modes(case)) * case.get("coils", 1) > 4e12


def exact(case, seed):
    if _too_long(case):
        return None
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batched":
        f_out, c_out = [], []
        for (M, n, _), x, c, f in zip(_problems(case), s["x"], s["c"], s["f"]):
            f_out.append(_direct1(x, c[None], n, 1)[0])
            c_out.append(_direct2(x, f[None], n, -1)[0][0])
        return f_out, c_out
    if kind == "type3":
        x, y = (v.double() for v in s["x"])
        u, v = (t.double() for t in s["t"])
        c = s["c"].to(torch.complex128)
        out = torch.empty(case["K"], dtype=torch.complex128, device=c.device)
        for a, b in _chunks(case["K"], case["M"]):
            ph = u[a:b, None] * x[None, :] + v[a:b, None] * y[None, :]
            out[a:b] = torch.polar(torch.ones((), device=c.device, dtype=torch.float64), ph) @ c
        return out
    xs, n = s["x"], _n_modes(case)
    if kind == "pair":
        return _direct1(xs, s["c"][None], n, 1)[0], _direct2(xs, s["f"][None], n, -1)[0][0]
    if kind == "normal":
        c = _direct2(xs, s["f"], n, -1)[0]
        return c, _direct1(xs, c, n, 1)
    if kind == "grad1":
        # L = sum |f - t|^2 with f = type 1: G = 2 (f - t), dL/dc_j = sum_k G_k e^{-i k x_j},
        # dL/dx_j = Re(conj(c_j) sum_k (-i k) G_k e^{-i k x_j})
        f = _direct1(xs, s["c"][None], n, 1)
        G = 2 * (f - s["f"][None])
        d = _direct2(xs, G, n, -1, grad=True)
        cc = s["c"].to(torch.complex128).conj()
        return (f[0], d[0][0], *[(cc * v[0]).real for v in d[1:]])
    # L = sum |c - d|^2 with c = type 2: G = 2 (c - d), dL/df_k = sum_j G_j e^{+i k x_j},
    # dL/dx_j = Re(conj(G_j) sum_k (-i k) f_k e^{-i k x_j})
    d = _direct2(xs, s["f"][None], n, -1, grad=True)
    G = 2 * (d[0] - s["c"][None])
    df = _direct1(xs, G, n, 1)
    return (d[0][0], df[0], *[(G[0].conj() * v[0]).real for v in d[1:]])

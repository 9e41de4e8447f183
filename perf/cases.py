"""The work this framework is used for, as timed cases: grid and point interpolation of a
particle snapshot, column-density images, neighbour searches and batches of snapshots, each
through the package's public entry points.

Every case is one snapshot of a seeded synthetic disc (the distributions of
``synthetic.disc`` and ``synthetic.clumped_disc``, made here on the GPU so that preparing is
quick) and one call, or the few calls, a user makes on it.  ``exact`` gives the same sums in
64 bits by plain dense evaluation, for the sizes where that is quick.
"""
import math

import numpy as np
import torch

import distorteddustydiscanalysistoolkits_b200 as pb
from distorteddustydiscanalysistoolkits_b200 import batch, synthetic

KERNELS = ("M4_spline", "M5_spline", "M6_spline", "C2_Wendland", "C4_Wendland", "C6_Wendland")
DENSE = 1.3e11     # particle-sample products up to which exact() evaluates densely


def listed():
    return [
        # a first look at a small snapshot: host arrays in and out, default precision; launches count
        dict(name="quicklook", kind="points", disc="disc", n=6000, grid="cartesian", n0=14, n1=14, n2=14,
             kernel="M4_spline", strategy="itpSymmetric", precision="fp64", fields="all", memory="host"),
        # the density of a gas disc on a Cartesian box (the first benchmark configuration)
        dict(name="density box", kind="points", disc="disc", n=131072, grid="cartesian", n0=64, n1=64, n2=64,
             kernel="M4_spline", strategy="itpSymmetric", precision="fp64", fields="rho", memory="host"),
        # all velocity derivatives on a cylindrical grid in the default precision
        dict(name="derivatives fp64", kind="points", disc="disc", n=400000, grid="cylindrical", n0=80, n1=80, n2=24,
             kernel="M4_spline", strategy="itpSymmetric", precision="fp64", fields="all", memory="device"),
        # the headline benchmark: 2^21 particles, 256 x 256 x 64 cylindrical grid, 11 outputs
        dict(name="derivatives fp32c", kind="points", disc="disc", n=2097152, grid="cylindrical", n0=256, n1=256,
             n2=64, kernel="M4_spline", strategy="itpSymmetric", precision="fp32c", fields="all", memory="device"),
        # a clumped disc with Wendland kernels: uneven work, density and vorticity
        dict(name="clumped vorticity", kind="points", disc="clumped", n=1048576, grid="cartesian", n0=96, n1=96,
             n2=96, kernel="C4_Wendland", strategy="itpSymmetric", precision="fp32c", fields="curl", memory="device"),
        # gather sums with a wide kernel on an odd grid
        dict(name="gather wide kernel", kind="points", disc="disc", n=250007, grid="cylindrical", n0=61, n1=83,
             n2=37, kernel="M6_spline", strategy="itpGather", precision="fp64", fields="rho_grad", memory="device"),
        # values at tracer positions, several sets of them on one tree that the program keeps
        dict(name="tracers on a tree", kind="tracers", disc="disc", n=300011, points=100003,
             kernel="C2_Wendland", strategy="itpScatter", precision="fp32c", fields="all", memory="device"),
        # a face-on column-density image
        dict(name="image face-on", kind="lines", disc="disc", n=1500000, n0=1024, n1=1024, view="face-on",
             kernel="M4_spline", precision="fp64", memory="device"),
        # a small oblique image from host arrays
        dict(name="image oblique", kind="lines", disc="disc", n=20011, n0=97, n1=61, view="oblique",
             kernel="M5_spline", precision="fp64", memory="host"),
        # a tree of a large snapshot and neighbour searches on it
        dict(name="tree and neighbours", kind="neighbours", disc="disc", n=4194304, points=20000, kernel="M4_spline"),
        # several snapshots of uneven size in one step (density and its gradient)
        dict(name="snapshot batch", kind="batch", n=250000, discs=4, n0=48, kernel="M4_spline",
             strategy="itpSymmetric", precision="fp32c", fields="rho_grad"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "points", "points", "tracers", "lines", "neighbours", "batch"])
    kernel = rng.choice(KERNELS)
    if kind == "neighbours":
        return dict(kind=kind, disc="disc", n=_log(rng, 6000, 4194304), points=_log(rng, 1000, 100000),
                    kernel=kernel)
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 30000, 250000), discs=rng.randint(2, 6), n0=rng.randint(12, 48),
                    kernel=kernel, strategy="itpSymmetric", precision=rng.choice(["fp64", "fp32c"]),
                    fields="rho_grad")
    memory = rng.choice(["host", "device"])
    if kind == "lines":
        return dict(kind=kind, disc="disc", n=_log(rng, 6000, 1500000), n0=_log(rng, 40, 1024),
                    n1=_log(rng, 40, 1024), view=rng.choice(["face-on", "oblique"]), kernel=kernel,
                    precision=rng.choice(["fp64", "fp32c"]), memory=memory)
    precision = rng.choice(["fp64", "fp32c"])
    case = dict(kind=kind, disc=rng.choice(["disc", "disc", "clumped"]), n=_log(rng, 6000, 2097152), kernel=kernel,
                strategy=rng.choice(["itpSymmetric", "itpSymmetric", "itpGather", "itpScatter"]),
                precision=precision, fields=rng.choice(["rho", "rho_grad", "curl", "all"]), memory=memory)
    # samples: at most what the largest listed case costs (FP64 and the wide kernels cost more)
    most = (4e12 if precision == "fp32c" else 5e11) / (4.0 if kernel in ("M5_spline", "M6_spline") else 1.0)
    points = _log(rng, 1000, max(2000, min(4.0e6, most / case["n"])))
    if kind == "tracers":
        case["points"] = points
        return case
    a = points ** (1.0 / 3.0)
    n0, n1 = max(4, int(a * rng.uniform(0.6, 1.6))), max(4, int(a * rng.uniform(0.6, 1.6)))
    case.update(grid=rng.choice(["cartesian", "cylindrical"]), n0=n0, n1=n1, n2=max(2, points // (n0 * n1)))
    return case


# ---- inputs ----
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Random:
    def __init__(self, seed):
        self.dev = _device()
        self.g = torch.Generator(device=self.dev).manual_seed(int(seed) * 7919 + 17)

    def uniform(self, lo, hi, *n):
        return lo + (hi - lo) * torch.rand(*n, generator=self.g, dtype=torch.float64, device=self.dev)

    def normal(self, *n):
        return torch.randn(*n, generator=self.g, dtype=torch.float64, device=self.dev)


def _particles(case, seed):
    """Columns of one snapshot: r ~ U[1, 100], H = 0.05 r^1.25, a warp, Keplerian velocities with
    1 % noise, h = 1.2 (m / rho)^(1/3); "clumped" adds two spiral arms and Gaussian clumps."""
    g, n = _Random(seed), case["n"]
    mass, rmin, rmax = 1e-6, 1.0, 100.0
    tilt = 15.0 if case["disc"] == "disc" else 30.0
    clumps = 0 if case["disc"] == "disc" else max(1, n // 8192)
    each = (n // 10) // clumps if clumps else 0
    nc = each * clumps
    nd = n - nc
    r = g.uniform(rmin, rmax, nd)
    phi = g.uniform(0.0, 2.0 * math.pi, nd)
    if clumps:   # two logarithmic arms, pitch 12 degrees: keep 1 in 5 of the samples far from an arm
        for _ in range(6):
            d = torch.remainder(phi - torch.log(r) / math.tan(math.radians(12.0)), math.pi)
            w = 0.2 + 0.8 * torch.exp(-torch.minimum(d, math.pi - d) ** 2 / 0.02)
            phi = torch.where(g.uniform(0.0, 1.0, nd) < w, phi, g.uniform(0.0, 2.0 * math.pi, nd))
    H = 0.05 * r ** 1.25
    zp = g.normal(nd) * H
    rho = (n * mass / (2.0 * math.pi * (rmax - rmin) * r)) / (math.sqrt(2.0 * math.pi) * H) * \
        torch.exp(-zp * zp / (2.0 * H * H))
    x, y = r * torch.cos(phi), r * torch.sin(phi)
    if clumps:
        at = (g.uniform(0.0, 1.0, clumps) * nd).long().clamp(max=nd - 1)
        size = torch.exp(g.uniform(math.log(0.05), math.log(0.5), clumps)) * H[at]
        off = g.normal(3, nc)
        s = size.repeat_interleave(each)
        rho = torch.cat([rho, each * mass / ((2.0 * math.pi) ** 1.5 * s ** 3) * torch.exp(-0.5 * (off ** 2).sum(0))])
        x, y, zp = (torch.cat([a, a[at].repeat_interleave(each) + o * s]) for a, o in zip((x, y, zp), off))
    rr = torch.sqrt(x * x + y * y)
    beta = math.radians(tilt) * (rr.clamp(rmin, rmax) - rmin) / (rmax - rmin)
    vk = rr.clamp(min=rmin) ** -0.5
    v = g.normal(3, n) * (0.01 * vk)
    vx, vy = -vk * y / rr, vk * x / rr
    c, s = torch.cos(beta), torch.sin(beta)
    return {"x": x, "y": y * c - zp * s, "z": y * s + zp * c, "m": torch.full_like(x, mass),
            "h": 1.2 * (mass / rho) ** (1.0 / 3.0), "rho": rho,
            "vx": vx + v[0], "vy": vy * c + v[1], "vz": vy * s + v[2]}


def _samples(case, p, seed):
    """Sample points (x, y, z): a box over the particles, a log-radius cylinder, or tracers near particles."""
    dev = p["x"].device
    if case["kind"] in ("tracers", "neighbours"):
        g = _Random(seed + 1000003)
        at = (g.uniform(0.0, 1.0, case["points"]) * case["n"]).long().clamp(max=case["n"] - 1)
        off = g.normal(3, case["points"]) * p["h"][at]
        return [(p[k][at] + o).contiguous() for k, o in zip("xyz", off)]
    n0, n1, n2 = case["n0"], case["n1"], case["n2"]
    lin = lambda a, b, k: torch.linspace(float(a), float(b), k, dtype=torch.float64, device=dev)   # noqa: E731
    if case["grid"] == "cartesian":
        axes = [lin(p[k].min(), p[k].max(), m) for k, m in zip("xyz", (n0, n1, n2))]
        c, b, a = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
        return [t.reshape(-1).contiguous() for t in (a, b, c)]
    hz = 3.0 * 0.05 * 100.0 ** 1.25
    c, b, a = torch.meshgrid(lin(-hz, hz, n2), torch.arange(n1, dtype=torch.float64, device=dev) * (2 * math.pi / n1),
                             torch.exp(lin(0.0, math.log(100.0), n0)), indexing="ij")
    return [t.reshape(-1).contiguous() for t in (a * torch.cos(b), a * torch.sin(b), c)]


def _lines(case, p):
    """Origins and unit directions of an image plane spanning the particles."""
    lo, hi = [min(float(p[k].min()) for k in "xy"), max(float(p[k].max()) for k in "xy")]
    lin = lambda k: torch.linspace(lo, hi, k, dtype=torch.float64, device=p["x"].device)   # noqa: E731
    b, a = torch.meshgrid(lin(case["n1"]), lin(case["n0"]), indexing="ij")
    a, b = a.reshape(-1), b.reshape(-1)
    t = 0.0 if case["view"] == "face-on" else math.radians(50.0)
    d = (0.0, -math.sin(t), math.cos(t))
    o = (a, b * math.cos(t), b * math.sin(t))
    return [c.contiguous() for c in o], [torch.full_like(a, c) for c in d]


_COLUMNS = {"rho": ("rho",), "rho_grad": ("rho",), "curl": ("rho", "vx", "vy", "vz"), "all": ("rho", "vx", "vy", "vz")}
_CATALOG = {"rho": dict(scalars=("rho",)), "rho_grad": dict(scalars=("rho",), gradients=("rho",)),
            "curl": dict(scalars=("rho",), curls=("v",)),
            "all": dict(scalars=("rho", "vx", "vy", "vz"), gradients=("rho",), divergences=("v",), curls=("v",))}
_L = {"rho": 1, "rho_grad": 4, "curl": 4, "all": 11}


def _batch_jobs(case, seed):
    jobs = []
    for k in range(case["discs"]):
        n = max(2000, int(case["n"] / 2.0 ** k) + 7 * k)
        p = synthetic.disc(n, seed=1000 * int(seed) + k, tilt_deg=10.0 * k)
        edge = max(6, case["n0"] - 7 * k)
        flat = pb.flatten(pb.Cartesian, synthetic.cartesian_box_grid(p, n=edge))
        inp = pb.InterpolationInput(p["x"], p["y"], p["z"], p["m"], p["h"], p["rho"], (p["rho"].copy(),),
                                    smoothed_kernel=getattr(pb, case["kernel"]))
        jobs.append({"input": inp, "points": flat,
                     "catalog": pb.InterpolationCatalog(("rho",), **_CATALOG[case["fields"]])})
    return jobs


def prepare(case, seed):
    if case["kind"] == "batch":
        # a program that steps through many sets of snapshots keeps the captured step
        db = batch.DeviceBatch(_batch_jobs(case, seed), precision=case["precision"],
                               strategy=getattr(pb, case["strategy"]))
        db.capture()
        return dict(case, db=db)
    p = _particles(case, seed)
    host = case.get("memory") == "host"
    put = (lambda t: t.cpu().numpy()) if host else (lambda t: t.contiguous())   # noqa: E731
    backend = pb.CUDAComputeBackend(0)
    state = dict(case, backend=backend)
    columns = ("rho", "vz") if case["kind"] == "lines" else _COLUMNS[case.get("fields", "rho")]
    state["input"] = pb.InterpolationInput(*[put(p[k]) for k in ("x", "y", "z", "m", "h", "rho")],
                                           tuple(put(p[k].clone()) for k in columns),
                                           smoothed_kernel=getattr(pb, case["kernel"]))
    if case["kind"] == "neighbours":
        state["points"] = [t.cpu().numpy() for t in _samples(case, p, seed)]
        state["radius"] = np.full(case["points"], 1.5 * float(p["h"].median()))
    elif case["kind"] == "lines":
        o, d = _lines(case, p)
        state["lines"] = pb.LineSamples(put(torch.zeros_like(o[0])), [put(t) for t in o], [put(t) for t in d])
        state["catalog"] = pb.InterpolationCatalog(columns, scalars=columns)
    else:
        q = [put(t) for t in _samples(case, p, seed)]
        state["catalog"] = pb.InterpolationCatalog(columns, **_CATALOG[case["fields"]])
        state["out"] = None if host else [torch.empty_like(q[0]) for _ in range(state["catalog"].L)]
        if case["kind"] == "tracers":
            state["points"] = q
            torch.cuda.synchronize()
            state["tree"] = pb.LinearBVH_build(state["input"], backend)
        else:
            state["samples"] = pb.PointSamples(np.zeros_like(q[0]) if host else torch.zeros_like(q[0]), q)
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["db"].replay()
        return state["db"].outs
    backend = state["backend"]
    if kind == "neighbours":
        tree = pb.LinearBVH_build(state["input"], backend, permute_input=False)
        nearest = pb.LBVH_find_nearest(tree, state["points"])
        return [nearest, *pb.LBVH_probe_neighbors(tree, state["points"], state["radius"])]
    if kind == "lines":
        grids = pb.LineSamples_interpolation(backend, state["lines"], state["input"], state["catalog"],
                                             pb.itpScatter, precision=state["precision"]).grids
        return [g.grid for g in grids]
    strategy = getattr(pb, state["strategy"])
    if kind == "tracers":
        return pb.interpolate_points(state["tree"], state["catalog"], state["points"], strategy,
                                     precision=state["precision"], out=state["out"])
    grids = pb.PointSamples_interpolation(backend, state["samples"], state["input"], state["catalog"], strategy,
                                          precision=state["precision"], out=state["out"]).grids
    return [g.grid for g in grids]


# ---- the necessary work and the 64-bit values ----
_VALID = {"M5_spline": 2.5, "M6_spline": 3.0}
_SIGMA = {"M4_spline": 1.0, "M5_spline": 0.05, "M6_spline": 1.0 / 120.0, "C2_Wendland": 21.0 / 16.0,
          "C4_Wendland": 495.0 / 256.0, "C6_Wendland": 1365.0 / 512.0}
_SPLINE = {"M4_spline": ((2.0, 0.25), (1.0, -1.0)), "M5_spline": ((2.5, 1.0), (1.5, -5.0), (0.5, 10.0)),
           "M6_spline": ((3.0, 1.0), (2.0, -6.0), (1.0, 15.0))}
_POWER = {"M4_spline": 3, "M5_spline": 4, "M6_spline": 5}
_WENDLAND = {"C2_Wendland": (4, (1.0, 2.0)), "C4_Wendland": (6, (1.0, 3.0, 35.0 / 12.0)),
             "C6_Wendland": (8, (1.0, 4.0, 6.25, 4.0))}


def _f(kernel, q):
    if kernel in _SPLINE:
        return sum(c * (a - q).clamp(min=0.0) ** _POWER[kernel] for a, c in _SPLINE[kernel])
    k, poly = _WENDLAND[kernel]
    return (1.0 - 0.5 * q).clamp(min=0.0) ** k * sum(c * q ** i for i, c in enumerate(poly))


def _df(kernel, q):
    if kernel in _SPLINE:
        k = _POWER[kernel]
        return sum(-k * c * (a - q).clamp(min=0.0) ** (k - 1) for a, c in _SPLINE[kernel])
    k, poly = _WENDLAND[kernel]
    t = (1.0 - 0.5 * q).clamp(min=0.0)
    return t ** k * sum(i * c * q ** (i - 1) for i, c in enumerate(poly) if i) - \
        0.5 * k * t ** (k - 1) * sum(c * q ** i for i, c in enumerate(poly))


def _radius2(case, p, ha):
    K = _VALID.get(case["kernel"], 2.0)
    ra, rb = (K * ha).square()[:, None], (K * p["h"]).square()[None]
    return torch.maximum(ra, rb) if case["strategy"] == "itpSymmetric" else ra if case["strategy"] == "itpGather" else rb


def _blocks(p, q, most=1.2e8):
    """(first sample, squared distances to every particle) by blocks of samples."""
    step = max(1, int(most / p["x"].numel()))
    for s in range(0, q[0].numel(), step):
        d2 = torch.zeros((min(step, q[0].numel() - s), p["x"].numel()), dtype=torch.float64, device=p["x"].device)
        for k, c in zip("xyz", q):
            d2 += (c[s:s + step, None] - p[k][None]).square_()
        yield s, d2


def _accepted(case):
    """Mean accepted neighbours of a sample, from a few hundred samples of one snapshot."""
    p = _particles(case, 1)
    if case["kind"] == "lines":
        o, d = _lines(case, p)
        at = torch.linspace(0, o[0].numel() - 1, 256, device=o[0].device).long()
        d2 = _line_d2(p, [c[at] for c in o], [c[at] for c in d])
        return float((d2 <= (_VALID.get(case["kernel"], 2.0) * p["h"]).square()[None]).sum()) / len(at)
    q = _samples(case, p, 1)
    at = torch.linspace(0, q[0].numel() - 1, 256, device=q[0].device).long()
    n = 0
    for _, d2 in _blocks(p, [c[at] for c in q]):
        n += int((d2 <= _radius2(case, p, p["h"][d2.argmin(1)])).sum())
    return n / len(at)


def work(case):
    """Bytes: every input column and sample read once, every output written once.  Operations:
    the accepted pairs (a mean over a few hundred samples) at the operations of one pair's terms."""
    if case["kind"] == "neighbours":
        n, m = case["n"], case["points"]
        return {"bytes": 7.0 * 8 * n + 8.0 * 8 * m, "flops": 60.0 * (n + 40.0 * m)}
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["discs"]):
            edge = max(6, case["n0"] - 7 * k)
            one = dict(case, kind="points", disc="disc", n=max(2000, int(case["n"] / 2.0 ** k) + 7 * k),
                       grid="cartesian", n0=edge, n1=edge, n2=edge)
            total = {key: total[key] + v for key, v in work(one).items()}
        return total
    if case["kind"] == "lines":
        m = case["n0"] * case["n1"]
        return {"bytes": 8.0 * (8 * case["n"] + 8 * m), "flops": 40.0 * m * _accepted(case)}
    m = case["points"] if case["kind"] == "tracers" else case["n0"] * case["n1"] * case["n2"]
    columns = 6 + len(_COLUMNS[case["fields"]])
    return {"bytes": 8.0 * (columns * case["n"] + (3 + _L[case["fields"]]) * m),
            "flops": {"rho": 45.0, "rho_grad": 80.0, "curl": 95.0, "all": 110.0}[case["fields"]] * m * _accepted(case)}


def _sums(values, counts):
    """Sums over consecutive segments of every row of `values`, in 64 bits."""
    return torch.stack([torch.segment_reduce(v, "sum", lengths=counts, initial=0.0) for v in values])


def _exact_points(case, p, q):
    kernel, strategy, fields = case["kernel"], case["strategy"], case["fields"]
    sigma = _SIGMA[kernel] / math.pi
    out = torch.empty((_L[fields], q[0].numel()), dtype=torch.float64, device=q[0].device)
    for s, d2 in _blocks(p, q):
        ha = p["h"][d2.argmin(1)]
        near = d2 <= _radius2(case, p, ha)
        counts = near.sum(1)
        i, b = near.nonzero(as_tuple=True)
        del near
        r = d2[i, b].sqrt()
        del d2
        W, G = torch.zeros_like(r), torch.zeros_like(r)
        sides = {"itpGather": (ha[i],), "itpScatter": (p["h"][b],)}.get(strategy, (ha[i], p["h"][b]))
        for h in sides:
            W += sigma / h ** 3 * _f(kernel, r / h) / len(sides)
            G += sigma / h ** 4 * _df(kernel, r / h) / len(sides)
        ml = p["m"][b] / p["rho"][b]
        a = [p[k][b] for k in _COLUMNS[fields]]
        w = ml * W
        G = ml * torch.where(r > 0, G / r, torch.zeros_like(r))
        g = [G * (c[s:s + len(ha)][i] - p[k][b]) for k, c in zip("xyz", q)]
        S = _sums(torch.stack([w] + [v * w for v in a]), counts)
        bar = [v / S[0] for v in S[1:]]
        rows = [S[1]] + (bar[1:] if fields == "all" else [])
        if fields != "rho":
            B = _sums(torch.stack(g), counts)
        if fields in ("rho_grad", "all"):
            F = _sums(torch.stack([v * a[0] for v in g]), counts)
            rows += [F[k] - bar[0] * B[k] for k in range(3)]
        if fields == "all":
            D = _sums((g[0] * a[1] + g[1] * a[2] + g[2] * a[3])[None], counts)[0]
            rows.append(D - (bar[1] * B[0] + bar[2] * B[1] + bar[3] * B[2]))
        if fields in ("curl", "all"):
            v = a[1:]
            for x, y in ((1, 2), (2, 0), (0, 1)):
                C = _sums((v[x] * g[y] - v[y] * g[x])[None], counts)[0]
                rows.append(-(C - (bar[1 + x] * B[y] - bar[1 + y] * B[x])))
        rows = torch.stack(rows)
        out[:, s:s + len(ha)] = torch.where(S[0] == 0.0, torch.full_like(rows, math.nan), rows)
    return list(out)


def _line_d2(p, o, d):
    D2 = torch.zeros((o[0].numel(), p["x"].numel()), dtype=torch.float64, device=p["x"].device)
    Dm = torch.zeros_like(D2)
    for k, a, m in zip("xyz", o, d):
        t = p[k][None] - a[:, None]
        D2 += t * t
        Dm += t * m[:, None]
    return D2 - Dm * Dm


def _column_table(kernel, dev, n=4096):
    """sigma * integral of f(sqrt(q^2 + s^2)) ds at n equally spaced q up to the support radius."""
    K = _VALID.get(kernel, 2.0)
    x, w = (torch.from_numpy(a).to(dev) for a in np.polynomial.legendre.leggauss(96))
    q = torch.linspace(0.0, K, n, dtype=torch.float64, device=dev)
    qs = q.clamp(min=1e-9)[:, None]
    ends = [0.0] + sorted(a for a, _ in _SPLINE.get(kernel, ((K, 0.0),)))
    at = [torch.acosh((torch.as_tensor(e, dtype=torch.float64, device=dev) / qs).clamp(min=1.0)) for e in ends]
    total = torch.zeros_like(q)
    for a, b in zip(at[:-1], at[1:]):   # s = q sinh t
        t = 0.5 * (b - a) * x + 0.5 * (b + a)
        r = qs * torch.cosh(t)
        total += (0.5 * (b - a) * w * 2.0 * r * _f(kernel, r)).sum(1)
    return total * _SIGMA[kernel] / math.pi, K


def _exact_lines(case, p, o, d):
    table, K = _column_table(case["kernel"], p["x"].device)
    step = max(1, int(4e7 / case["n"]))
    out = [torch.empty_like(o[0]) for _ in range(2)]
    for s in range(0, o[0].numel(), step):
        d2 = _line_d2(p, [c[s:s + step] for c in o], [c[s:s + step] for c in d])
        near = d2 <= (K * p["h"]).square()[None]
        u = (d2.clamp(min=0.0).sqrt() / p["h"] / K * 4095.0).clamp(max=4095.0)
        k = u.long().clamp(max=4094)
        t = u - k
        w = torch.where(near, (table[k] * (1.0 - t) + table[k + 1] * t) / p["h"] * p["m"] / p["rho"],
                        torch.zeros_like(u))
        S = w.sum(1)
        none = torch.full_like(S, math.nan)
        out[0][s:s + step] = torch.where(S == 0.0, none, w @ p["rho"])
        out[1][s:s + step] = torch.where(S == 0.0, none, (w @ p["vz"]) / S)
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        if case["discs"] * case["n"] * case["n0"] ** 3 > 3.0 * DENSE:
            return None
        out = []
        for job in _batch_jobs(case, seed):
            t = lambda a: torch.from_numpy(np.array(a)).to(_device())   # noqa: E731
            i = job["input"]
            p = dict(zip(("x", "y", "z", "m", "h", "rho"), (t(a) for a in (*i.coord, i.m, i.h, i.rho))))
            out.append(_exact_points(case, p, [t(a) for a in job["points"].coor]))
        return out
    p = _particles(case, seed)
    if case["kind"] == "lines":
        if 1.0 * case["n"] * case["n0"] * case["n1"] > DENSE:
            return None
        return _exact_lines(case, p, *_lines(case, p))
    q = _samples(case, p, seed)
    if 1.0 * case["n"] * q[0].numel() > DENSE:
        return None
    if case["kind"] == "neighbours":
        d2 = torch.cat([b.amin(1) for _, b in _blocks(p, q)])
        return [None, None, None, torch.where(d2 <= (1.5 * float(p["h"].median())) ** 2, d2,
                                              torch.full_like(d2, math.inf))]
    return _exact_points(case, p, q)

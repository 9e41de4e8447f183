"""Particles with a negative smoothing length (accreted ones that a program has not dropped) against the CPU
oracle, bit for bit: a leaf's own radius may then exceed its subtree's, so which leaves are reached depends
on every node above them, for points and for lines."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
import oracle

pytestmark = pytest.mark.gpu


def _cloud(n, h, many):
    """A few (or every tenth) of the particles with h = -20 times the others'."""
    g = np.random.default_rng(n)
    p = {k: g.uniform(-1.0, 1.0, n) for k in "xyz"}
    p.update(h=h * g.uniform(0.2, 1.8, n), m=np.ones(n), rho=g.uniform(0.5, 2.0, n))
    at = slice(None, None, 10) if many else [1, n // 2]
    p["h"][at] = -20.0 * p["h"][at]
    return p


def _input(p):
    return pb.InterpolationInput(*[p[k].copy() for k in ("x", "y", "z", "m", "h", "rho")], (p["rho"].copy(),),
                                 smoothed_kernel=pb.M4_spline)


def _equal(got, exp):
    assert np.array_equal(np.isnan(got), np.isnan(exp))
    ok = ~np.isnan(exp)
    assert np.array_equal(got[ok], exp[ok])


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("n", [2, 16, 17, 40, 3000])
@pytest.mark.parametrize("strategy", ["itpSymmetric", "itpGather", "itpScatter"])
def test_points(backend, n, many, strategy):
    p = _cloud(n, 0.05, many)
    g = np.random.default_rng(1)
    q = [g.uniform(-1.2, 1.2, 500) for _ in "xyz"]
    cat = pb.InterpolationCatalog(("rho",), scalars=("rho",))
    o = oracle.OracleLBVH(p["x"], p["y"], p["z"], p["h"]).attach(p["m"], p["rho"], [p["rho"]], "M4_spline")
    exp, st = o.interp_points(cat.oracle_dict(), *q, strategy=strategy, stats=True)
    out = pb.PointSamples_interpolation(backend, pb.PointSamples(np.zeros(500), q), _input(p), cat,
                                        getattr(pb, strategy), precision=pb.FP64)
    assert sum(backend.handle.pair_split()[2:]) == int(st[:, 4].sum())   # accepted pairs
    _equal(out.grids[0].grid, exp[0])


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("n,lines", [(2, 60), (40, 60), (3000, 60), (400, 131072)])
def test_lines(backend, n, lines, many):
    """131,072 lines are the first to be taken by tiles."""
    p = _cloud(n, 0.05, many)
    a = np.linspace(-1.1, 1.1, lines if lines < 1000 else 512)
    a, b = [c.ravel() for c in np.meshgrid(a, np.linspace(-1.0, 1.0, lines // len(a)))]
    t = np.radians(35.0)
    o = [a, b * np.cos(t), b * np.sin(t)]
    d = [np.zeros(lines), np.full(lines, -np.sin(t)), np.full(lines, np.cos(t))]
    cat = pb.InterpolationCatalog(("rho",), scalars=("rho",))
    ref = oracle.OracleLBVH(p["x"], p["y"], p["z"], p["h"]).attach(p["m"], p["rho"], [p["rho"]], "M4_spline")
    out = pb.LineSamples_interpolation(backend, pb.LineSamples(np.zeros(lines), o, d), _input(p), cat, pb.itpScatter)
    _equal(out.grids[0].grid, ref.interp_lines(cat.oracle_dict(), o, d)[0])

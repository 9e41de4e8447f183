"""FP64 sums around the count from which a block instead of a warp takes a query (the size class above 1,024:
1,280 accepted leaves) against the CPU oracle, bit for bit, for every catalog shape and strategy and a wide
kernel, and with queries on both sides of it in one launch."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
import oracle

pytestmark = pytest.mark.gpu

COLS = ("rho", "vx", "vy", "vz")
CATALOGS = {"scalar": dict(scalars=("rho",)), "scalar + gradient": dict(scalars=("rho",), gradients=("rho",)),
            "curl": dict(scalars=("rho", "vy"), curls=("v",)),
            "all": dict(scalars=COLS, gradients=("rho",), divergences=("v",), curls=("v",)),
            "two scalars": dict(scalars=("rho", "vx"))}


def _cloud(n, h, shift=0.0):
    g = np.random.default_rng(n)
    p = {k: g.normal(0.0, 1.0, n) + shift for k in "xyz"}
    p.update({k: g.normal(0.0, 1.0, n) for k in ("vx", "vy", "vz")})
    p["h"], p["m"], p["rho"] = h * g.uniform(0.5, 1.5, n), g.uniform(0.5, 2.0, n), g.uniform(0.1, 3.0, n)
    return p


def _same(p, q, catalog, strategy, kernel, backend):
    inp = pb.InterpolationInput(*[p[k].copy() for k in ("x", "y", "z", "m", "h", "rho")], tuple(p[c].copy() for c in COLS),
                                smoothed_kernel=getattr(pb, kernel))
    cat = pb.InterpolationCatalog(COLS, **catalog)
    out = pb.PointSamples_interpolation(backend, pb.PointSamples(np.zeros(len(q[0])), q), inp, cat, getattr(pb, strategy),
                                        precision=pb.FP64)
    got = np.stack([g.grid for g in out.grids])
    o = oracle.OracleLBVH(p["x"], p["y"], p["z"], p["h"]).attach(p["m"], p["rho"], [p[c] for c in COLS], kernel)
    exp, st = o.interp_points(cat.oracle_dict(), *q, strategy=strategy, stats=True)
    assert not np.isnan(exp).any() and np.array_equal(got, exp)
    return st[:, 4]


@pytest.mark.parametrize("strategy,kernel", [("itpSymmetric", "M4_spline"), ("itpGather", "M6_spline"),
                                             ("itpScatter", "C4_Wendland")])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 1279, 1280, 1281, 1311, 1312, 1375, 1376, 1377])
def test_counts(backend, n, strategy, kernel):
    q = [np.random.default_rng(5).normal(0.0, 1.0, 3) for _ in "xyz"]
    p = _cloud(n, 20.0)
    for name in CATALOGS:
        assert (_same(p, q, CATALOGS[name], strategy, kernel, backend) == n).all()


@pytest.mark.parametrize("strategy", ["itpSymmetric", "itpGather", "itpScatter"])
def test_both_forms_in_one_launch(backend, strategy):
    """A cloud of 1,400 and, out of reach, one of 300: of 40 queries 14 go to blocks."""
    a, b = _cloud(1400, 20.0), _cloud(300, 20.0, 1000.0)
    p = {k: np.concatenate([a[k], b[k]]) for k in a}
    q = [np.random.default_rng(6).normal(0.0, 1.0, 40) + np.where(np.arange(40) % 3, 1000.0, 0.0) for _ in "xyz"]
    for name in CATALOGS:
        count = _same(p, q, CATALOGS[name], strategy, "M4_spline", backend)
        assert sorted(set(count)) == [300, 1400] and (count == 1400).sum() == 14

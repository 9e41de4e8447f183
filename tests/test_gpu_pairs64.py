"""The FP64 pair kernels' branches against the CPU oracle, bit for bit: every catalog shape a
launch is specialised for, query sizes around the 32-lane batches and around the point where a
block instead of a warp sums a query, and particles outside the range of the short divisions."""
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


def _cloud(n, seed, h):
    g = np.random.default_rng(seed)
    p = {k: g.normal(0.0, 1.0, n) for k in ("x", "y", "z")}
    p.update({k: g.normal(0.0, 1.0, n) for k in ("vx", "vy", "vz")})
    p["h"], p["m"], p["rho"] = h * g.uniform(0.5, 1.5, n), g.uniform(0.5, 2.0, n), g.uniform(0.1, 3.0, n)
    return p


def _same(p, q, catalog, strategy, kernel, backend):
    columns = COLS if any(k in catalog for k in ("divergences", "curls")) or len(catalog["scalars"]) > 1 else ("rho",)
    inp = pb.InterpolationInput(*[p[k].copy() for k in ("x", "y", "z", "m", "h", "rho")],
                                tuple(p[c].copy() for c in columns), smoothed_kernel=getattr(pb, kernel))
    cat = pb.InterpolationCatalog(columns, **catalog)
    flat = pb.PointSamples(np.zeros(len(q[0])), q)
    out = pb.PointSamples_interpolation(backend, flat, inp, cat, getattr(pb, strategy), precision=pb.FP64)
    got = np.stack([g.grid for g in out.grids])
    o = oracle.OracleLBVH(p["x"], p["y"], p["z"], p["h"]).attach(p["m"], p["rho"], [p[c] for c in columns], kernel)
    exp = o.interp_points(cat.oracle_dict(), *q, strategy=strategy)
    assert np.array_equal(np.isnan(got), np.isnan(exp))
    ok = ~np.isnan(exp)
    assert np.array_equal(got[ok], exp[ok])


@pytest.mark.parametrize("catalog", sorted(CATALOGS))
@pytest.mark.parametrize("kernel", ["M4_spline", "M5_spline", "M6_spline", "C2_Wendland", "C4_Wendland", "C6_Wendland"])
def test_every_catalog_shape(backend, catalog, kernel):
    """Points inside, at the edge of and outside the supports, on a particle, and far away."""
    p = _cloud(900, 3, 0.4)
    g = np.random.default_rng(4)
    q = [np.concatenate([g.normal(0.0, 1.5, 150), p[k][:20], [40.0]]) for k in "xyz"]
    for strategy in ("itpSymmetric", "itpGather", "itpScatter"):
        _same(p, q, CATALOGS[catalog], strategy, kernel, backend)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 95, 96, 97, 8191, 8192, 8193, 8289])
def test_batch_and_block_edges(backend, n):
    """Every particle accepted by every point: counts at the edges of the batches, of the block form's
    rounds (three batches) and of the count from which a block takes the query."""
    p = _cloud(n, n, 20.0)
    g = np.random.default_rng(5)
    q = [g.normal(0.0, 1.0, 3) for _ in "xyz"]
    for name in ("scalar", "all"):
        _same(p, q, CATALOGS[name], "itpSymmetric", "M4_spline", backend)


@pytest.mark.parametrize("what", ["h", "rho", "m"])
def test_particles_outside_the_short_divisions(backend, what):
    """One particle whose h, rho or m is extreme, zero or negative sends the pairs to the general
    divisions."""
    for value in (1e-90, 0.0, -0.5) if what != "h" else (1e-90, -0.5):
        p = _cloud(300, 8, 0.5)
        p[what][7] = value
        q = [np.concatenate([np.random.default_rng(9).normal(0.0, 1.0, 60), p[k][5:9]]) for k in "xyz"]
        for strategy in ("itpSymmetric", "itpScatter"):
            with np.errstate(all="ignore"):
                _same(p, q, CATALOGS["all"], strategy, "M4_spline", backend)

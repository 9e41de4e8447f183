"""The walk of the two-phase point path against the CPU oracle's neighbour counts and sums: queries whose
runs fill one chunk, one extent and several, subtrees around the scanned size, deep trees, and the run
lists of a small pool."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
import oracle

pytestmark = pytest.mark.gpu


def _same(p, q, strategy, backend, kernel="M4_spline"):
    inp = pb.InterpolationInput(*[p[k].copy() for k in ("x", "y", "z", "m", "h", "rho")], (p["rho"].copy(),),
                                smoothed_kernel=getattr(pb, kernel))
    cat = pb.InterpolationCatalog(("rho",), scalars=("rho",))
    out = pb.PointSamples_interpolation(backend, pb.PointSamples(np.zeros(len(q[0])), q), inp, cat,
                                        getattr(pb, strategy), precision=pb.FP64)
    got = out.grids[0].grid
    o = oracle.OracleLBVH(p["x"], p["y"], p["z"], p["h"]).attach(p["m"], p["rho"], [p["rho"]], kernel)
    exp, st = o.interp_points(cat.oracle_dict(), *q, strategy=strategy, stats=True)
    assert sum(backend.handle.pair_split()[2:]) == int(st[:, 4].sum())   # accepted pairs
    assert np.array_equal(np.isnan(got), np.isnan(exp[0]))
    ok = ~np.isnan(exp[0])
    assert np.array_equal(got[ok], exp[0][ok])


def _lattice(n, h):
    g = np.random.default_rng(n)
    p = {k: g.uniform(-1.0, 1.0, n) for k in "xyz"}
    p.update(h=h * g.uniform(0.2, 1.8, n), m=np.ones(n), rho=g.uniform(0.5, 2.0, n))
    return p


@pytest.mark.parametrize("strategy", ["itpSymmetric", "itpGather", "itpScatter"])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 18, 33, 512, 5000])
def test_small_trees(backend, n, strategy):
    p = _lattice(n, 0.3)
    g = np.random.default_rng(1)
    _same(p, [np.concatenate([g.uniform(-1.5, 1.5, 200), p[k][:5]]) for k in "xyz"], strategy, backend)


@pytest.mark.parametrize("strategy", ["itpSymmetric", "itpScatter"])
def test_many_runs_per_query(backend, strategy):
    """Supports that vary by 10 make accepted and rejected leaves alternate: up to thousands of runs a
    query, over several extents."""
    p = _lattice(60000, 0.35)
    p["h"] = 0.35 * np.random.default_rng(2).choice([0.1, 1.0], 60000)
    g = np.random.default_rng(3)
    _same(p, [g.uniform(-1.0, 1.0, 60) for _ in "xyz"], strategy, backend)


def test_deep_tree(backend):
    p = _lattice(4000, 0.2)
    for k in "xyz":
        p[k][:3000] = 0.125
    g = np.random.default_rng(4)
    q = [np.concatenate([g.uniform(-1.0, 1.0, 50), np.full(3, 0.125)]) for _ in "xyz"]
    for strategy in ("itpSymmetric", "itpGather", "itpScatter"):
        _same(p, q, strategy, backend)


@pytest.mark.parametrize("chunks", ["7", "8", "15", "64"])
def test_pools_of_a_few_extents(monkeypatch, chunks):
    """A pool that holds no whole extent (7), one (8, 15) or eight of them: the queries go through in
    rounds or by the fused kernels, with the same values."""
    monkeypatch.setenv("PB_RUN_POOL_CHUNKS", chunks)
    be = pb.CUDAComputeBackend(0)
    try:
        p = _lattice(3000, 0.3)
        g = np.random.default_rng(5)
        _same(p, [g.uniform(-1.2, 1.2, 300) for _ in "xyz"], "itpSymmetric", be)
    finally:
        be.close()

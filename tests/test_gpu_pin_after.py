"""The staging of small host arrays in ordinary memory (page-locked memory refused or not yet due), and where it
becomes page-locked between the calls and within one: the same outputs and in-place order."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
from distorteddustydiscanalysistoolkits_b200 import synthetic

pytestmark = pytest.mark.gpu


def _calls(be):
    """A growing and a shrinking set of host arrays: points, lines and neighbours."""
    out = []
    for n, m in ((300, 20), (5000, 900), (1000, 30)):
        p = synthetic.disc(n, seed=4)
        cols = [p[k].copy() for k in ("x", "y", "z", "m", "h", "rho", "vx")]
        inp = pb.InterpolationInput(*cols[:6], (cols[6],))
        g = np.random.default_rng(n)
        q = [g.uniform(-90.0, 90.0, m), g.uniform(-90.0, 90.0, m), g.normal(0.0, 3.0, m)]
        cat = pb.InterpolationCatalog(("v",), scalars=("v",))
        res = pb.PointSamples_interpolation(be, pb.PointSamples(np.zeros(m), q), inp, cat, pb.itpSymmetric)
        out += [res.grids[0].grid, *cols]
        d = [np.zeros(m), np.zeros(m), np.ones(m)]
        out.append(pb.LineSamples_interpolation(be, pb.LineSamples(np.zeros(m), q, d), inp, cat, pb.itpScatter).grids[0].grid)
        out.append(pb.LBVH_find_nearest_h(pb.LinearBVH(be, n), q))
    return out


@pytest.mark.parametrize("after", [0, 1, 2, 3, 4, 7, 32])
def test_same_bits(backend, after):
    ref = _calls(backend)
    be = pb.CUDAComputeBackend(0)
    try:
        be.handle.set_option("pin_after", after)
        got = _calls(be)
    finally:
        be.close()
    for a, b in zip(got, ref):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


def test_option_range(backend):
    for value in (-1, 1 << 31):
        with pytest.raises(pb.ArgumentError):
            backend.handle.set_option("pin_after", value)


# 16,384 particles, points or lines are the last to be packed in ordinary memory, 32,768 in page-locked memory
@pytest.mark.parametrize("after", [0, 1])
@pytest.mark.parametrize("n", [16384, 16385, 32768, 32769])
def test_largest_arrays(after, n):
    p = synthetic.disc(n, seed=4)
    g = np.random.default_rng(n)
    q = [g.uniform(-90.0, 90.0, n), g.uniform(-90.0, 90.0, n), g.normal(0.0, 3.0, n)]
    cat = pb.InterpolationCatalog(("v",), scalars=("v",))
    got = []
    for option in (after, 0):
        be = pb.CUDAComputeBackend(0)
        try:
            be.handle.set_option("pin_after", option)
            for _ in range(2):
                cols = [p[k].copy() for k in ("x", "y", "z", "m", "h", "rho", "vx")]
                inp = pb.InterpolationInput(*cols[:6], (cols[6],))
                grids = pb.PointSamples_interpolation(be, pb.PointSamples(np.zeros(n), q), inp, cat, pb.itpGather).grids
                d = [np.zeros(n), np.zeros(n), np.ones(n)]
                lines = pb.LineSamples_interpolation(be, pb.LineSamples(np.zeros(n), q, d), inp, cat, pb.itpScatter).grids
                got.append([grids[0].grid, lines[0].grid, *cols])
        finally:
            be.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64))

"""The list of long walks, used up to 7 in 8 of the queries and not beyond: the same outputs as in the plain order,
for sets whose share on the list is none, all, and just below and above that, in one slice and in several."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 2000, 40001])   # a warp and a thread per nearest search
@pytest.mark.parametrize("long", [0.0, 0.49, 0.85, 0.9, 1.0])
def test_same_bits(backend, m, long):
    g = np.random.default_rng(m)
    n = 3000
    x = np.sort(g.uniform(0.0, 1.0, (3, n)), axis=1)
    h = np.where(x[0] < long, 0.08, 0.004)      # the particles of small x are 20 times as wide
    if long == 0.0:
        h[:3] = 1.0                             # three wide particles: hardly a query has one as its nearest
    inp = pb.InterpolationInput(*x, np.ones(n), h, g.uniform(0.5, 2.0, n), (g.normal(0.0, 1.0, n),), smoothed_kernel=pb.M4_spline)
    tree = pb.LinearBVH_build(inp, backend)
    cat = pb.InterpolationCatalog(("a",), scalars=("a",))
    u = g.uniform(0.0, 1.0, m)
    q = [u + 0.01 * g.normal(size=m) for _ in "xyz"]   # near the particles' diagonal: x tells which are long
    out = []
    for schedule, slice_queries in ((0, 1 << 22), (1, 1 << 22), (1, 1024)):
        backend.handle.set_option("schedule", schedule)
        backend.handle.set_option("slice_queries", slice_queries)
        for strategy in (pb.itpSymmetric, pb.itpGather):
            out.append(pb.interpolate_points(tree, cat, q, strategy, precision=pb.FP64)[0])
            out.append(np.array(backend.handle.pair_split(), np.float64))
    backend.handle.set_option("schedule", 1)
    backend.handle.set_option("slice_queries", 1 << 22)
    for k in range(4, len(out)):
        assert np.array_equal(out[k].view(np.uint64), out[k % 4].view(np.uint64))

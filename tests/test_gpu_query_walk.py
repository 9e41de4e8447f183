"""The warp walk of the neighbour queries against brute force: whole subtrees inside the radius, radii of
zero, infinity and NaN, points on particles and equal distances, tiny and deep trees."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 16, 17, 40, 3000])
def test_query_and_probe_match_brute_force(backend, n):
    g = np.random.default_rng(n)
    x = g.integers(0, 12, (3, n)) / 4.0   # a lattice: duplicates and equal distances
    one = np.ones(n)
    tree = pb.LinearBVH_build(pb.InterpolationInput(*[c.copy() for c in x], one.copy(), one.copy(), one.copy(), ()),
                              backend, permute_input=False)
    order = tree.encoding()[1]
    s = x[:, order]
    q = np.concatenate([g.uniform(-1.0, 4.0, (3, 60)), x[:, :20], [[1e30], [0.0], [0.0]]], axis=1)
    m = q.shape[1]
    r = g.choice([0.0, 0.25, 0.8, 2.0, 30.0, np.inf, np.nan], m)
    with np.errstate(all="ignore"):
        d2 = (q[0][:, None] - s[0]) ** 2 + (q[1][:, None] - s[1]) ** 2 + (q[2][:, None] - s[2]) ** 2
        hit = d2 <= (r * r)[:, None]
    best = np.where(hit & (d2 < np.inf), d2, np.inf)
    idx = np.where(np.isfinite(best.min(1)), best.argmin(1), -1)
    count, near, near_d2 = pb.LBVH_probe_neighbors(tree, q, r)
    assert np.array_equal(count, hit.sum(1))
    assert np.array_equal(near, idx) and np.array_equal(near_d2, best.min(1))
    for i, sel in enumerate(pb.LBVH_query(tree, q, r)):
        assert np.array_equal(sel.valid_indices(), np.flatnonzero(hit[i])) and sel.nearest == idx[i]

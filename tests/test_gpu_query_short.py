"""Many neighbour queries (24,576 and more): short walks are finished by a thread each, the others by a warp
each.  Radii on both sides of that, none and all of the leaves, both ends of the size rule, and a pool that
is too small."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 40, 3000])
@pytest.mark.parametrize("m", [24575, 24576, 33000])
def test_counts_lists_and_closest(backend, n, m):
    g = np.random.default_rng(n)
    x = g.integers(0, 12, (3, n)) / 4.0   # equal positions and distances
    one = np.ones(n)
    tree = pb.LinearBVH_build(pb.InterpolationInput(*[c.copy() for c in x], one.copy(), one.copy(), one.copy(), ()),
                              backend, permute_input=False)
    s = x[:, tree.encoding()[1]]
    q = np.concatenate([g.uniform(-1.0, 4.0, (3, 60)), x[:, :20], [[1e30], [0.0], [0.0]]], axis=1)
    k = q.shape[1]
    r = g.choice([0.0, 0.25, 0.8, 2.0, 30.0, np.inf, np.nan], k)
    with np.errstate(all="ignore"):
        d2 = (q[0][:, None] - s[0]) ** 2 + (q[1][:, None] - s[1]) ** 2 + (q[2][:, None] - s[2]) ** 2
        hit = d2 <= (r * r)[:, None]
    near = np.where(hit & (d2 < np.inf), d2, np.inf)
    best = near.min(1)
    idx = np.where(np.isfinite(best), near.argmin(1), -1)
    at = np.arange(m) % k
    got = pb.LBVH_probe_neighbors(tree, q[:, at], r[at])
    assert np.array_equal(got[0], hit.sum(1)[at]) and np.array_equal(got[1], idx[at])
    assert np.array_equal(got[2], best[at])
    sel = pb.LBVH_query(tree, q[:, at], r[at])
    for i in (*range(k), *range(m - k, m)):
        assert np.array_equal(sel[i].valid_indices(), np.flatnonzero(hit[at[i]])) and sel[i].nearest == idx[at[i]]


def test_pool_too_small(backend):
    """A list that does not fit is reported and nothing is written past its end, by either form."""
    n, m = 500, 24576
    g = np.random.default_rng(3)
    x = g.random((3, n))
    one = np.ones(n)
    tree = pb.LinearBVH_build(pb.InterpolationInput(*[c.copy() for c in x], one.copy(), one.copy(), one.copy(), ()), backend)
    q = np.ascontiguousarray(x[:, np.arange(m) % n])
    H, P = tree.handle, pb._lib.ptr
    for radius in (0.05, 5.0):
        r = np.full(m, radius)
        off = np.arange(m + 1, dtype=np.int64)   # one place each
        off[1:] -= 1                             # and none for the first
        pool = np.full(m, -7, np.int64)
        near = np.empty(m, np.int64)
        with pytest.raises(pb.DimensionMismatch):
            H.check(H.lib.pb_query_neighbors(H.h, m, P(q[0]), P(q[1]), P(q[2]), P(r), P(off), P(pool), P(near)), "query")


@pytest.mark.parametrize("m", [100, 24576])
def test_empty_lists_fit_any_offsets(backend, m):
    """Offsets that go back are refused only for a query that has something to write."""
    g = np.random.default_rng(4)
    x = g.random((3, 300))
    one = np.ones(300)
    tree = pb.LinearBVH_build(pb.InterpolationInput(*[c.copy() for c in x], one.copy(), one.copy(), one.copy(), ()), backend)
    q = g.uniform(5.0, 6.0, (3, m))   # nothing within 0.1
    off = np.arange(m + 1, dtype=np.int64) % 3
    off[-1] = 0
    r, pool, near = np.full(m, 0.1), np.full(4, -7, np.int64), np.empty(m, np.int64)
    H, P = tree.handle, pb._lib.ptr
    H.check(H.lib.pb_query_neighbors(H.h, m, P(q[0]), P(q[1]), P(q[2]), P(r), P(off), P(pool), P(near)), "query")
    assert (near == -1).all() and (pool == -7).all()

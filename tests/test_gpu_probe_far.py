"""The closest leaf of a probe is searched within its radius only: leaves exactly at the radius, points with
nothing inside it, and points so far away that FP32 boxes do not tell distances apart, by a warp each (up
to 32,768 points) and by a thread each."""
import time

import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb

pytestmark = pytest.mark.gpu


def _tree(x, backend):
    one = np.ones(x.shape[1])
    tree = pb.LinearBVH_build(pb.InterpolationInput(*[c.copy() for c in x], one.copy(), one.copy(), one.copy(), ()),
                              backend, permute_input=False)
    return tree, x[:, tree.encoding()[1]]


@pytest.mark.parametrize("n", [1, 2, 33, 700])
@pytest.mark.parametrize("copies", [1, 200])
def test_matches_brute_force(backend, n, copies):
    g = np.random.default_rng(n)
    tree, s = _tree(g.integers(0, 9, (3, n)) / 4.0, backend)
    q = np.concatenate([g.integers(-8, 24, (3, 150)) / 4.0, g.normal(0.0, 1.0, (3, 50)) * 10.0 ** g.integers(0, 31, 50)], axis=1)
    d2 = ((q[0][:, None] - s[0]) ** 2 + (q[1][:, None] - s[1]) ** 2) + (q[2][:, None] - s[2]) ** 2
    r = g.choice([0.0, 0.25, 0.5, 1.25, 4.0, 1e9, 1e25, 1e200, np.inf, np.nan], 200)   # many d2 equal r^2 on the lattice
    with np.errstate(over="ignore", invalid="ignore"):
        near = np.where((d2 <= (r * r)[:, None]) & (d2 < np.inf), d2, np.inf)
    best = near.min(1)
    idx = np.where(best < np.inf, near.argmin(1), -1)
    got = pb.LBVH_probe_neighbors(tree, np.tile(q, (1, copies)), np.tile(r, copies))
    assert np.array_equal(got[1], np.tile(idx, copies)) and np.array_equal(got[2], np.tile(best, copies))


@pytest.mark.parametrize("m", [2000, 40000])
def test_far_points_cost_no_more(backend, m):
    g = np.random.default_rng(7)
    tree, _ = _tree(g.normal(0.0, 50.0, (3, 200000)), backend)
    ms = []
    for scale in (50.0, 1e9, 1e30):
        q = g.normal(0.0, scale, (3, m))
        t = []
        for _ in range(10):
            a = time.perf_counter()
            pb.LBVH_probe_neighbors(tree, q, 1.0)
            t.append(time.perf_counter() - a)
        ms.append(min(t[1:]))
    assert max(ms[1:]) < 8.0 * ms[0]

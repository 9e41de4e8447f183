"""The warp's nearest search (up to 32,768 points) against the thread's (above) and brute force: ties,
points outside the particles' box and beyond FP32, flat axes, tiny trees."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65, 5000])
@pytest.mark.parametrize("kind", ["lattice", "flat", "random"])
def test_matches_brute_force_and_the_thread_search(backend, n, kind):
    g = np.random.default_rng(n)
    x = g.integers(0, 9, (3, n)) / 4.0 if kind == "lattice" else g.normal(0.0, 1.0, (3, n))
    if kind == "flat":
        x[2] = 0.75
    one = np.ones(n)
    tree = pb.LinearBVH_build(pb.InterpolationInput(*[c.copy() for c in x], one.copy(), one.copy(), one.copy(), ()),
                              backend, permute_input=False)
    s = x[:, tree.encoding()[1]]
    q = np.concatenate([g.uniform(-3.0, 5.0, (3, 200)), g.integers(-2, 11, (3, 200)) / 8.0, x[:, :50],
                        [[1e30, -1e25, 0.0], [0.0, 1e24, 1e5], [0.0, 0.0, -1e6]]], axis=1)
    d2 = ((q[0][:, None] - s[0]) ** 2 + (q[1][:, None] - s[1]) ** 2) + (q[2][:, None] - s[2]) ** 2
    got = pb.LBVH_find_nearest(tree, q)
    assert np.array_equal(got, d2.argmin(1))
    many = np.tile(q, (1, 32768 // q.shape[1] + 1))   # more than 32,768 points: a thread each
    assert np.array_equal(pb.LBVH_find_nearest(tree, many), np.tile(got, 32768 // q.shape[1] + 1))

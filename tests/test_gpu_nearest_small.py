"""The nearest search of few particles: up to 12,288 (below 512 particles), 24,576 (below 4,096) and 32,768 points by a
warp each, above by a thread each, with the same results against brute force on both sides."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,limit", [(511, 12288), (512, 24576), (4095, 24576), (4096, 32768)])
def test_both_sides(backend, n, limit):
    g = np.random.default_rng(n)
    x = g.integers(0, 30, (3, n)) / 4.0   # equal positions and distances
    one = np.ones(n)
    h = g.uniform(0.5, 1.0, n)
    tree = pb.LinearBVH_build(pb.InterpolationInput(*[c.copy() for c in x], one.copy(), h, one.copy(), ()), backend)
    s = np.stack([x[:, i] for i in tree.encoding()[1]], axis=1)
    q = np.concatenate([g.uniform(-1.0, 9.0, (3, 150)), g.integers(0, 60, (3, 150)) / 8.0], axis=1)
    d2 = ((q[0][:, None] - s[0]) ** 2 + (q[1][:, None] - s[1]) ** 2) + (q[2][:, None] - s[2]) ** 2
    exp = d2.argmin(1)
    for m in (limit, limit + 1):
        at = np.arange(m) % 300
        assert np.array_equal(pb.LBVH_find_nearest(tree, q[:, at]), exp[at])
        assert np.array_equal(pb.LBVH_find_nearest_h(tree, q[:, at]), h[exp[at]])   # h is in tree order by now

"""Tiles of lines that lie far apart (across a jump of the Morton order, or with origins at scattered depths) go
line by line in a launch of their own: the values are those of a warp per line, and such an image does
not take longer than a larger regular one."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
from distorteddustydiscanalysistoolkits_b200 import synthetic

pytestmark = pytest.mark.gpu


def _image(edge, depth):
    a, b = [c.ravel() for c in np.meshgrid(np.linspace(-90.0, 90.0, edge), np.linspace(-90.0, 90.0, edge))]
    z = np.random.default_rng(1).uniform(-depth, depth, a.size) if depth else np.zeros(a.size)
    return [a, b, z], [np.zeros(a.size), np.zeros(a.size), np.ones(a.size)]


@pytest.fixture(scope="module")
def tree(backend):
    p = synthetic.disc(1500000, seed=13)
    inp = pb.InterpolationInput(p["x"], p["y"], p["z"], p["m"], p["h"], p["rho"], (p["rho"].copy(), p["vz"]),
                                smoothed_kernel=pb.M5_spline)
    return pb.LinearBVH_build(inp, backend)


CAT = pb.InterpolationCatalog(("rho", "vz"), scalars=("rho", "vz"))


@pytest.mark.parametrize("depth", [0.0, 300.0])
def test_values(tree, depth):
    """363^2 lines are above the 131,072 from which tiles are taken, half of them below."""
    o, d = _image(363, depth)
    got = np.stack(pb.interpolate_lines(tree, CAT, o, d))
    at = np.random.default_rng(2).permutation(363 * 363)[:60000]
    exp = np.stack(pb.interpolate_lines(tree, CAT, [c[at] for c in o], [c[at] for c in d]))
    assert np.array_equal(got[:, at].view(np.uint64), exp.view(np.uint64))


@pytest.mark.parametrize("edge,depth", [(363, 0.0), (400, 300.0)])
def test_time(tree, edge, depth):
    H = tree.handle
    H.set_option("timing", 1)
    ms = []
    for o, d in (_image(edge, depth), _image(512, 0.0)):
        for _ in range(8):
            pb.interpolate_lines(tree, CAT, o, d)
            ms.append(H.timings()[1])
    H.set_option("timing", 0)
    assert min(ms[1:8]) < 2.5 * min(ms[9:])

"""The line kernels' branches against the CPU oracle, bit for bit: a warp per line and tiles of 32 lines
(from 131,072 lines on), images along and across the axes, tiles whose lines differ in direction or
share few particles, ragged counts, tiny and degenerate trees."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
import oracle

pytestmark = pytest.mark.gpu


def _cloud(n, h, seed=1):
    g = np.random.default_rng(seed)
    p = {k: g.normal(0.0, 1.0, n) for k in ("x", "y", "z", "vz")}
    p["h"], p["m"], p["rho"] = h * g.uniform(0.3, 1.7, n), g.uniform(0.5, 2.0, n), g.uniform(0.1, 3.0, n)
    return p


def _image(n0, n1, direction, half=2.5):
    d = np.asarray(direction, float) / np.linalg.norm(direction)
    e1 = np.cross(d, (0.3, 1.0, 0.2)) if abs(d[1]) < 0.9 else np.array([1.0, 0.0, 0.0])
    e1 -= d * (e1 @ d)
    e1 /= np.linalg.norm(e1)
    e2 = np.cross(d, e1)
    a, b = np.meshgrid(np.linspace(-half, half, n0), np.linspace(-half, half, n1), indexing="ij")
    a, b = a.ravel(), b.ravel()
    return [a * e1[k] + b * e2[k] + 0.7 * d[k] for k in range(3)], [np.full(a.shape, d[k]) for k in range(3)]


def _check(backend, p, o, d, kernel="M4_spline", precision=pb.FP64):
    cols = ("rho", "vz")
    inp = pb.InterpolationInput(*[p[k].copy() for k in ("x", "y", "z", "m", "h", "rho")],
                                tuple(p[c].copy() for c in cols), smoothed_kernel=getattr(pb, kernel))
    cat = pb.InterpolationCatalog(cols, scalars=cols)
    out = pb.LineSamples_interpolation(backend, pb.LineSamples(np.zeros(len(o[0])), o, d), inp, cat, pb.itpScatter,
                                       precision=precision)
    got = np.stack([g.grid for g in out.grids])
    ref = oracle.OracleLBVH(p["x"], p["y"], p["z"], p["h"]).attach(p["m"], p["rho"], [p[c] for c in cols], kernel)
    exp = ref.interp_lines(cat.oracle_dict(), o, d)
    assert np.array_equal(np.isnan(got), np.isnan(exp))
    ok = ~np.isnan(exp)
    assert np.array_equal(got[ok], exp[ok])


@pytest.mark.parametrize("n,h", [(1, 1.0), (2, 1.0), (33, 0.5), (700, 0.15)])
@pytest.mark.parametrize("shape", [(1, 1), (31, 1), (33, 3), (363, 362)])
@pytest.mark.parametrize("direction", [(0, 0, 1), (0, 1, 0), (0.2, -0.5, 0.8)])
def test_images(backend, n, h, shape, direction):
    """363 x 362 lines are 4,106 tiles, the last one of 6 lines."""
    _check(backend, _cloud(n, h), *_image(*shape, direction))


@pytest.mark.parametrize("kernel", ["M5_spline", "M6_spline", "C6_Wendland"])
def test_kernels_and_precisions(backend, kernel):
    p = _cloud(400, 0.2)
    for precision in (pb.FP64, pb.FP32C):
        _check(backend, p, *_image(365, 360, (0, 0, 1)), kernel=kernel, precision=precision)


@pytest.mark.parametrize("count", [777, 131072])
def test_directions_differ_within_a_tile(backend, count):
    """A pinhole view (one origin) and random directions: no tile has one direction."""
    g = np.random.default_rng(3)
    p = _cloud(300, 0.1)
    d = g.normal(size=(3, count))
    d /= np.linalg.norm(d, axis=0)
    _check(backend, p, [np.full(count, c) for c in (0.1, -4.0, 0.3)], list(d))
    _check(backend, p, [g.normal(0.0, 2.0, count) for _ in range(3)], list(d))


def test_tiles_that_share_few_particles(backend):
    """Supports far smaller than a tile: after the probe the lines are taken one by one."""
    _check(backend, _cloud(60000, 0.004), *_image(512, 257, (0, 0, 1)))


def test_slightly_longer_direction(backend):
    """|d| = 1 + 1e-9 keeps the general node bound."""
    o, d = _image(20, 25, (0.2, -0.5, 0.8))
    _check(backend, _cloud(300, 0.2), o, [c * (1.0 + 1e-9) for c in d])


def test_deep_tree(backend):
    """Equal positions: the duplicate bump makes a tree of long chains."""
    p = _cloud(3000, 0.2)
    for k in ("x", "y", "z"):
        p[k][:2500] = 0.25
    _check(backend, p, *_image(40, 40, (0, 0, 1)))

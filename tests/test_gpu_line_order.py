"""Line tiles taken by their estimated work (from 262,144 particles and 131,072 lines on) against the CPU
oracle, bit for bit: one direction, and tiles of mixed directions among them; a ragged last tile."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [262143, 262144])
@pytest.mark.parametrize("mixed", [False, True])
def test_ordered_tiles(backend, n, mixed):
    g = np.random.default_rng(n)
    r = np.exp(g.normal(-1.0, 1.0, n))   # dense in the middle
    a = g.uniform(0.0, 2.0 * np.pi, n)
    x, y, z = r * np.cos(a), r * np.sin(a), 0.1 * r * g.normal(0.0, 1.0, n)
    m, h, rho = g.uniform(0.5, 2.0, n), 0.01 * r * g.uniform(0.5, 1.5, n), g.uniform(0.1, 3.0, n)
    u, v = np.meshgrid(np.linspace(-2.0, 2.0, 363), np.linspace(-2.0, 2.0, 362), indexing="ij")
    o = [u.ravel(), v.ravel(), np.full(u.size, 0.3)]
    d = [np.zeros(u.size), np.zeros(u.size), np.ones(u.size)]
    if mixed:
        d[0][::997], d[2][::997] = 0.6, 0.8
    cat = pb.InterpolationCatalog(("rho",), scalars=("rho",))
    inp = pb.InterpolationInput(*[c.copy() for c in (x, y, z, m, h, rho)], (rho.copy(),), smoothed_kernel=pb.M4_spline)
    out = pb.LineSamples_interpolation(backend, pb.LineSamples(np.zeros(u.size), o, d), inp, cat, pb.itpScatter,
                                       precision=pb.FP64)
    got = np.stack([k.grid for k in out.grids])
    ref = oracle.OracleLBVH(x, y, z, h).attach(m, rho, [rho], "M4_spline")
    assert np.array_equal(got, ref.interp_lines(cat.oracle_dict(), o, d), equal_nan=True)

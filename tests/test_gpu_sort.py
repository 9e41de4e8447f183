"""The build's radix sort at the edges of its tiles (3,072 keys) and look-back, for uniform, clustered,
sorted and equal codes: order and codes against the CPU oracle."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 3071, 3072, 3073, 6143, 6144, 6145, 98304, 98305, 700001])
@pytest.mark.parametrize("kind", ["uniform", "clustered", "sorted", "equal"])
def test_order_and_codes(backend, n, kind):
    g = np.random.default_rng(n)
    x = g.random((3, n))
    if kind == "clustered":
        x[:, 1:] = 0.5 + 1e-5 * x[:, 1:]
    elif kind == "sorted":
        x = np.sort(x, axis=1)
    elif kind == "equal":
        x[:] = x[:, :1]
    h = np.full(n, 0.1)
    o = oracle.OracleLBVH(*x, h)
    codes, order = pb.MortonEncoding(*x, h, backend=backend)
    assert np.array_equal(order, o.order) and np.array_equal(codes, o.codes)


def test_pair_order_of_many_sizes(backend):
    """Counts over many size classes around the FP32C split: every query's value, whatever the order."""
    g = np.random.default_rng(1)
    n = 9000
    p = {k: g.normal(0.0, 1.0, n) for k in "xyz"}
    h = 10.0 ** g.uniform(-2.0, 0.3, n)
    rho, one = g.uniform(0.5, 2.0, n), np.ones(n)
    q = [g.normal(0.0, 1.0, 4097) for _ in "xyz"]
    cat = pb.InterpolationCatalog(("rho",), scalars=("rho",))
    out = {}
    for sched in (0, 1):
        backend.handle.set_option("schedule", sched)
        inp = pb.InterpolationInput(p["x"].copy(), p["y"].copy(), p["z"].copy(), one.copy(), h.copy(), rho.copy(), (rho.copy(),))
        out[sched] = pb.PointSamples_interpolation(backend, pb.PointSamples(np.zeros(4097), q), inp, cat, pb.itpSymmetric,
                                                   precision=pb.FP32C).grids[0].grid
        split = backend.handle.pair_split()
        assert split[0] > 0 and split[1] > 0 and split[0] + split[1] == 4097
    backend.handle.set_option("schedule", 1)
    assert np.array_equal(out[0].view(np.uint64), out[1].view(np.uint64))

"""A radix-sort tile that does not wait for the tiles before it counts their keys itself: codes, order and the
orders of the queries and pairs are the same (no read of them can meet a place that was not written)."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1])
def hasty(request):
    be = pb.CUDAComputeBackend(0)
    be.handle.set_option("sort_wait", request.param)
    yield be
    be.close()


@pytest.mark.parametrize("n", [2, 3072, 3073, 9217, 300001])
@pytest.mark.parametrize("kind", ["uniform", "clustered"])
def test_order_and_codes(hasty, n, kind):
    g = np.random.default_rng(n)
    x = g.random((3, n))
    if kind == "clustered":
        x[:, 1:] = 0.5 + 1e-5 * x[:, 1:]
    h = np.full(n, 0.1)
    o = oracle.OracleLBVH(*x, h)
    codes, order = pb.MortonEncoding(*x, h, backend=hasty)
    assert np.array_equal(order, o.order) and np.array_equal(codes, o.codes)


def test_interpolation(hasty, backend):
    g = np.random.default_rng(1)
    n, m = 20000, 30000
    p = {k: g.normal(0.0, 1.0, n) for k in "xyz"}
    q = [g.normal(0.0, 1.0, m) for _ in "xyz"]
    h, rho = 10.0 ** g.uniform(-2.0, -0.5, n), g.uniform(0.5, 2.0, n)
    cat = pb.InterpolationCatalog(("rho",), scalars=("rho",), gradients=("rho",))
    out = []
    for be in (hasty, backend):
        inp = pb.InterpolationInput(p["x"].copy(), p["y"].copy(), p["z"].copy(), np.ones(n), h.copy(), rho.copy(), (rho.copy(),))
        grids = pb.PointSamples_interpolation(be, pb.PointSamples(np.zeros(m), q), inp, cat, pb.itpSymmetric).grids
        out.append(np.stack([a.grid for a in grids]))
    assert np.array_equal(out[0].view(np.uint64), out[1].view(np.uint64))


def test_option_range(backend):
    for value in (-1, 1 << 31):
        with pytest.raises(pb.ArgumentError):
            backend.handle.set_option("sort_wait", value)

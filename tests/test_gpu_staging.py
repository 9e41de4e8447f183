"""Host arrays through the packed staging (2 MiB in all) and beyond it: outputs and the in-place order equal
those of device arrays, for points and lines, and a bad input leaves the caller's arrays alone."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
from distorteddustydiscanalysistoolkits_b200 import synthetic

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "z", "m", "h", "rho")


def _inputs(n, device):
    import torch
    p = synthetic.disc(n, seed=4)
    put = (lambda a: torch.from_numpy(a.copy()).cuda()) if device else (lambda a: a.copy())   # noqa: E731
    return pb.InterpolationInput(*[put(p[k]) for k in NAMES], (put(p["vx"]),)), p


def _host(a):
    return a.cpu().numpy() if hasattr(a, "cpu") else a


# seven columns of 8 bytes: 37,449 particles are the last to go packed; 87,381 points' three columns likewise
@pytest.mark.parametrize("n,points", [(500, 33), (37449, 87381), (37450, 87382)])
def test_points_host_and_device(backend, n, points):
    g = np.random.default_rng(1)
    q = [g.uniform(-90.0, 90.0, points), g.uniform(-90.0, 90.0, points), g.normal(0.0, 3.0, points)]
    cat = pb.InterpolationCatalog(("v",), scalars=("v",), gradients=("v",))
    got = []
    for device in (False, True):
        inp, _ = _inputs(n, device)
        out = pb.PointSamples_interpolation(backend, pb.PointSamples(np.zeros(points), q), inp, cat, pb.itpGather)
        got.append([o.grid for o in out.grids] + [_host(c) for c in (*inp.coord, inp.m, inp.h, inp.rho, *inp.quant)])
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("lines", [1, 43690, 43691])   # six columns: 43,690 lines are the last to go packed
def test_lines_host_and_device(backend, lines):
    import torch
    g = np.random.default_rng(2)
    o = [g.uniform(-90.0, 90.0, lines) for _ in range(2)] + [np.zeros(lines)]
    d = [np.zeros(lines), np.zeros(lines), np.ones(lines)]
    cat = pb.InterpolationCatalog(("v",), scalars=("v",))
    got = []
    for put in (lambda a: a, lambda a: torch.from_numpy(a).cuda()):
        inp, _ = _inputs(3000, False)
        ln = pb.LineSamples(put(np.zeros(lines)), [put(c) for c in o], [put(c) for c in d])
        got.append(_host(pb.LineSamples_interpolation(backend, ln, inp, cat, pb.itpScatter).grids[0].grid))
    assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64))


def test_rejected_input_is_left_alone(backend):
    inp, p = _inputs(500, False)
    inp.coord[1][7] = np.nan
    before = [c.copy() for c in (*inp.coord, inp.m, inp.h, inp.rho)]
    with pytest.raises(pb.ArgumentError):
        pb.LinearBVH_build(inp, backend)
    for a, b in zip(before, (*inp.coord, inp.m, inp.h, inp.rho)):
        assert np.array_equal(a, b, equal_nan=True)

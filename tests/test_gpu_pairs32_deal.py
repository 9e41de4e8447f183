"""FP32C pair sums dealt to blocks, four queries each (many queries, ordered by size class), and to warps (few
queries, or the plain order): the same bits on both sides of the rule (four queries a resident warp)."""
import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", [pb.itpSymmetric, pb.itpScatter])
def test_same_bits(backend, strategy):
    import torch
    resident = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    g = np.random.default_rng(1)
    n = 400
    p = {k: g.normal(0.0, 1.0, n) for k in "xyz"}
    inp = pb.InterpolationInput(p["x"], p["y"], p["z"], g.uniform(0.5, 2.0, n), 10.0 ** g.uniform(0.7, 1.3, n),
                                g.uniform(0.1, 3.0, n), (g.normal(0.0, 1.0, n),), smoothed_kernel=pb.M4_spline)
    tree = pb.LinearBVH_build(inp, backend)
    cat = pb.InterpolationCatalog(("a",), scalars=("a",), gradients=("a",))
    # 5 blocks of 4 warps an SM are meant; around 4 to 6 of them and a few queries past each
    edges = sorted({4 * resident * b + d for b in (4, 5, 6) for d in (-1, 0, 1, 3)})
    q = [g.normal(0.0, 1.0, edges[-1]) for _ in "xyz"]
    H = backend.handle
    H.set_option("fp64_light_max", 0)
    try:
        H.set_option("schedule", 0)
        plain = np.stack(pb.interpolate_points(tree, cat, q, strategy, precision=pb.FP32C))
        assert H.pair_split()[0] == edges[-1]   # every query on the FP32C kernel
        H.set_option("schedule", 1)
        for m in edges:
            got = np.stack(pb.interpolate_points(tree, cat, [c[:m] for c in q], strategy, precision=pb.FP32C))
            assert np.array_equal(got.view(np.uint64), plain[:, :m].view(np.uint64)), m
    finally:
        H.set_option("schedule", 1)
        H.set_option("fp64_light_max", 4096)

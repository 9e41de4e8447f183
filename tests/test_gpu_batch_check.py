"""pb_batch_check on asynchronous builds whose handles keep streams of their own: it waits for every one of them
and names the disc whose input was bad."""
import ctypes

import numpy as np
import pytest

import distorteddustydiscanalysistoolkits_b200 as pb
from distorteddustydiscanalysistoolkits_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [None, 0, 2])
@pytest.mark.parametrize("shared", [False, True])
def test_own_and_shared_streams(bad, shared):
    import torch
    g = np.random.default_rng(1)
    stream = torch.cuda.Stream()
    backends = [pb.CUDAComputeBackend(0) for _ in range(3)]
    keep = []
    try:
        for k, be in enumerate(backends):
            if shared:
                be.handle.set_stream(stream.cuda_stream)
            n = 200000 + 1000 * k
            x = g.random((3, n))
            if bad == k:
                x[1, n // 2] = np.nan
            cols = [torch.from_numpy(c).cuda() for c in x] + [torch.ones(n, dtype=torch.float64, device="cuda") for _ in range(3)]
            inp = pb.InterpolationInput(*cols, ())
            torch.cuda.synchronize()
            cin = inp._c_struct()
            keep.append((inp, cin))
            be.handle.check(be.handle.lib.pb_linear_bvh(be.handle.h, ctypes.byref(cin), _lib.PB_BUILD_ASYNC), "build")
        H = backends[0].handle
        handles = (ctypes.c_void_p * 3)(*[b.handle.h.value for b in backends])
        rc = H.lib.pb_batch_check(handles, 3)
        if bad is None:
            H.check(rc, "check")
        else:
            with pytest.raises(pb.ArgumentError, match="disc %d" % bad):
                H.check(rc, "check")
    finally:
        torch.cuda.synchronize()
        for be in backends:
            be.close()

"""A CUDA call that fails on the host is reported once: by the call that made it,
not by the next good one.  The failure is a stream capture that the library's own
synchronise invalidates; a launch into it is refused by the runtime, so nothing
reaches the GPU."""
import ctypes

import numpy as np
import pytest

from rapidfem_b200 import _native
from rapidfem_b200 import gpu as G
from rapidfem_b200 import operator as O

pytestmark = pytest.mark.gpu


def _runtime():
    import torch  # loads the CUDA runtime library
    assert torch.cuda.is_available()
    return torch, ctypes.CDLL("libcudart.so.12")


@pytest.mark.parametrize("engine", [_native.ENGINE_TF32X3, _native.ENGINE_FP32], ids=["tf32x3", "fp32"])
def test_a_refused_launch_does_not_fail_the_next_call(engine):
    torch, rt = _runtime()
    stream = torch.cuda.Stream()
    handle = ctypes.c_void_p(stream.cuda_stream)
    ctx = G.GpuContext(0)
    gop = G.GpuOperator(ctx, O.MaxwellOperator(O.structured_box(2, 2, 2), 3, 1.0))
    gop.set_engine(engine)
    y = np.random.default_rng(0).standard_normal(gop.n_dof()).astype(np.float32)
    want = gop.apply(y)
    gop.upload(y)
    ctx.set_stream(stream.cuda_stream)
    relaxed = 2
    assert rt.cudaStreamBeginCapture(handle, relaxed) == 0
    try:
        with pytest.raises(_native.DgtdError):
            ctx.synchronize()  # not allowed in a capture: invalidates it
        with pytest.raises(_native.DgtdError):
            gop.run_lserk(1e-3, 1)  # the launch is refused
    finally:
        graph = ctypes.c_void_p()
        assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) != 0
        rt.cudaGetLastError()
    gop.upload(y)
    gop.run_lserk(1e-3, 1)
    gop.download()
    assert np.array_equal(gop.apply(y), want)
    ctx.set_stream(None)

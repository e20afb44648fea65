"""A call that fails inside the CUDA runtime is reported by that call alone.

The library's copy of the runtime keeps the last error until it is read, and launches ask for it; an
error that a call has already reported must not come back from the next one.
"""

import ctypes as ct

import pytest
import torch

import azeban_b200 as az
from tests.gpu_helpers import VISC_CFGS, random_field_hat, to_dev

pytestmark = pytest.mark.gpu

RELAXED = 2  # CU_STREAM_CAPTURE_MODE_RELAXED


def test_failed_call_leaves_no_error_behind():
    """SSP_RK3.integrate waits for its stream, which a stream that is being captured refuses (and which
    ends the capture).  The transform after it succeeds, and so does the next step."""
    g = az.Grid(2, 16)
    ts = az.SSP_RK3(az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["smooth"], g)))
    u = to_dev(random_field_hat(2, 16, seed=5))
    ts.integrate(0.0, 1.0, 0.2, u)
    x = torch.randn((2, 16, 16), device="cuda", dtype=torch.float64)
    h = torch.empty((2, 16, 9), device="cuda", dtype=torch.complex128)
    fft = az.make_fft(h, x, az.FFT_FORWARD)
    fft.forward()
    stream = torch.cuda.Stream()
    cuda = ct.CDLL("libcuda.so.1")
    handle, graph = ct.c_void_p(stream.cuda_stream), ct.c_void_p()
    torch.cuda.synchronize()
    assert cuda.cuStreamBeginCapture_v2(handle, RELAXED) == 0
    with pytest.raises(az.AzebanError):
        ts.integrate(0.0, 1.0, 0.2, u, stream=stream)
    cuda.cuStreamEndCapture(handle, ct.byref(graph))  # the capture has ended already, without a graph
    fft.forward()
    assert torch.allclose(h, torch.fft.rfftn(x, dim=(1, 2)))
    assert ts.integrate(0.0, 1.0, 0.2, u) > 0.0

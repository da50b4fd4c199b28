"""A launch that fails is reported by the call that made it, and by no later one. The failure is made on
the host: a stream whose capture has been invalidated refuses launches."""
import ctypes

import pytest

import kernels_gb300 as kg
from kernels_gb300 import _lib

pytestmark = pytest.mark.gpu


def refused_stream(torch, stream):
    """Begin a capture on `stream` (through the driver, whose errors are no runtime error) and invalidate it."""
    driver = ctypes.CDLL("libcuda.so.1")
    handle = ctypes.c_void_p(stream.cuda_stream)
    assert driver.cuStreamBeginCapture_v2(handle, 1) == 0  # thread-local mode
    assert driver.cuStreamSynchronize(handle) == 900  # not permitted while capturing: the capture is invalid now

    def end():
        graph = ctypes.c_void_p()
        driver.cuStreamEndCapture(handle, ctypes.byref(graph))
    return end


@pytest.mark.parametrize("n", [64, 63])
def test_a_failed_launch_is_reported_once(cuda, n):
    in_a, in_b, out = kg.alloc(n)
    kg.init(in_a, out)
    kg.apply(kg.STAR, 2, in_a, out, in_b)
    cuda.cuda.synchronize()
    stream = cuda.cuda.Stream()
    for call in (lambda: kg.add(in_a, stream=stream), lambda: kg.apply(kg.STAR, 2, in_a, out, in_b, stream=stream),
                 lambda: kg.apply(kg.STAR, 2, in_a, out, stream=stream)):
        end = refused_stream(cuda, stream)
        try:
            with pytest.raises(kg.PrkError):
                call()
        finally:
            end()
        kg.init(in_a, out)  # <<<>>> and the last error: launches, and succeeds
    kg.add(in_a, stream=stream)
    cuda.cuda.synchronize()
    assert _lib.load().prk_gb300_status() == 0
    assert float(in_a[0, 0]) == 1.0

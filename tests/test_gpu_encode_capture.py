"""A code's first device encoding while the calling thread captures a stream: encoding was a
call that touches no stream of the caller's, and leaves the capture intact."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, 1])  # synchronising with the legacy stream, and not
def test_first_encode_inside_a_capture(cb, O, flags):
    rt = cb.lib()
    if not hasattr(rt, "cudaStreamBeginCapture"):
        pytest.skip("the CUDA runtime is not reachable through the library")
    code = cb.NrLdpc(704, 2112, base_graph=1, lifting_size=32, precision="f32")
    u = np.random.default_rng(3).integers(0, 2, (64, 704)).astype(np.uint8)  # above 2^15 lifted edges
    assert 64 * code.edges >= 1 << 15
    stream, graph = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(stream), flags) == 0
    assert rt.cudaStreamBeginCapture(stream, 0) == 0  # the global mode
    got = code.encode(u)
    assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0
    assert rt.cudaGraphDestroy(graph) == 0 and rt.cudaStreamDestroy(stream) == 0
    ref = O.Code(704, 2112, bg=1, z=32)
    for f in (0, 31, 63):
        assert np.array_equal(got[f], ref.encode(u[f]))

"""cb_encode in several chunks of the device buffer, and in a process forked after the device
was used: byte for byte the oracle's blocks."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = 128 << 20  # bytes of a chunk (capi.cu)


@pytest.mark.parametrize("k, e, bg, z", [(520, 1040, 2, 52), (520, 1041, 2, 52), (8448, 25344, 1, 384)])
def test_chunks_of_the_device_buffer(cb, O, k, e, bg, z):
    code = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f32")
    ref = O.Code(k, e, bg=bg, z=z)
    per = CHUNK // (k + e)
    n = 2 * per + 37  # a shorter last chunk
    u = np.random.default_rng(k + e).integers(0, 2, (n, k)).astype(np.uint8)
    got = code.encode(u)
    for f in sorted({0, 1, per - 1, per, per + 1, 2 * per - 1, 2 * per, n - 1}):
        assert np.array_equal(got[f], ref.encode(u[f])), f
    # the kept buffer holds a smaller call
    assert np.array_equal(code.encode(u[:300]), got[:300])


def test_a_forked_process_encodes_on_the_host(cb):
    code = cb.NrLdpc(8448, 25344, base_graph=1, lifting_size=384, precision="f32")
    u = np.random.default_rng(4).integers(0, 2, (2, 8448)).astype(np.uint8)
    want = code.encode(u)  # on the device
    pid = os.fork()
    if pid == 0:
        os._exit(0 if np.array_equal(code.encode(u), want) else 1)
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0
    assert np.array_equal(code.encode(u), want)

"""Blocks encoded on the device (csrc/encode.cu) against the oracle's encoder, byte for byte:
liftings that fill a word and that do not, filler bits, odd sent lengths (byte stores),
redundancy versions, the bit interleaver, repeated bits, bytes whose bit 0 alone counts, and
batches on both sides of the line from which the device encodes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(k=8448, e=25344, bg=1, z=384), dict(k=8400, e=12675, bg=1, z=384), dict(k=520, e=1040, bg=2, z=52),
    dict(k=20, e=77, bg=2, z=2), dict(k=22 * 32, e=1501, bg=1, z=32), dict(k=333, e=1200, bg=2, z=36, rv=3, qm=6),
    dict(k=640, e=8000, bg=2, z=64, rv=2, qm=2)])
def test_device_encoder_equals_the_oracle(cb, O, kw):
    kw = dict(kw)
    k, e, bg, z = (kw.pop(x) for x in ("k", "e", "bg", "z"))
    code = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f32", **kw)
    ref = O.Code(k, e, bg=bg, z=z, **kw)
    rng = np.random.default_rng(k)
    # the device encodes from 2^15 lifted edges on
    line = -(-(1 << 15) // code.edges)
    for n in sorted({1, max(1, line - 1), line, line + 3}):
        u = rng.integers(0, 256, (n, k)).astype(np.uint8)
        got = code.encode(u)
        for f in sorted({0, n // 2, n - 1}):
            assert np.array_equal(got[f], ref.encode(u[f] & 1)), (n, f)

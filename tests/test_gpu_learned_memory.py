"""Device memory of the training passes: the row records, and message gradients of less than twice
the lifted edges, at a lifting just above a stride of the backward kernels."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shared", [True, False])
def test_gradients_take_what_their_edges_need(cb, shared):
    import torch

    z, T, n = 72, 2, 512
    k, e = 10 * z, 20 * z
    code = cb.NrLdpc(k, e, base_graph=2, lifting_size=z, precision="f32")
    net = cb.LearnedNms(code, T, shared=shared)
    rng = np.random.default_rng(0)
    llr = rng.standard_normal((n, e)).astype(np.float32)
    cw = np.zeros((n, code.n_full), np.uint8)
    net.gradients(llr[:1], cw[:1])  # the code's own buffers and the kernels
    before = torch.cuda.mem_get_info()[0]
    net.gradients(llr, cw)
    used = before - torch.cuda.mem_get_info()[0]
    records = 12 * code.n_rows * T
    gradients = 2 * 4 * code.edges
    words = 4 * (e + code.n_full * (1 + T)) + code.n_full * 2 + 64
    assert used <= n * (records + gradients + words) + 8 * (4 << 20)  # (allocations come in pages)

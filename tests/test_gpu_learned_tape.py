"""The training kernels' row records and warp sums (csrc/nms_learned.cu) against the oracle's
forward and adjoint in the same f32 arithmetic: both base graphs (rows of 3 to 19 edges), liftings
of one partial warp, of a warp and an odd remainder and of the largest block, weights shared
and per lifted edge, one and several frames, one and several iterations."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bg, z, n, T", [(1, 2, 3, 3), (1, 7, 5, 2), (2, 3, 1, 1), (2, 32, 4, 3), (1, 44, 3, 2),
                                         (1, 384, 2, 2)])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("multi", [0, 2])
def test_records_and_sums_equal_the_oracle(cb, O, bg, z, n, T, shared, multi):
    k, e = (22 if bg == 1 else 10) * z, (44 if bg == 1 else 20) * z
    g = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f32")
    ref = O.Code(k, e, bg=bg, z=z)
    net = cb.LearnedNms(g, T, shared=shared)
    rng = np.random.default_rng(z)
    alpha = (0.75 + 0.05 * rng.standard_normal(net.n_weights)).astype(np.float32)
    beta = (0.05 * np.abs(rng.standard_normal(net.n_weights))).astype(np.float32)
    net.set_weights(alpha, beta)
    cw = np.stack([ref.encode_full(u) for u in rng.integers(0, 2, (n, k)).astype(np.uint8)])
    sent = cw[:, 2 * z:2 * z + e]
    llr = (2.0 * (1.0 - 2.0 * sent) + 2.0 * rng.standard_normal((n, e))).astype(np.float32)
    loss, ga, gb = net.gradients(llr, cw, multi_loss=multi)
    rloss, rpost, (rga, rgb) = ref.learned(T, shared, alpha, beta, llr, cw, want_post=True, want_grad=True,
                                           multi=multi, precision="f32")
    assert np.array_equal(net.forward(llr).view(np.uint32), rpost.view(np.uint32))
    # the bounds of tests/test_gpu_learned.py: the order of the f32 sums and CUDA's expf
    assert abs(loss - rloss) <= 1e-5 * abs(rloss)
    for got, want in ((ga, rga), (gb, rgb)):
        assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("bg, z, cols", [(1, 20, 44), (1, 20, 25), (2, 52, 20), (2, 36, 12)])
@pytest.mark.parametrize("low", [0.0, -0.05])
@pytest.mark.parametrize("multi, info_only", [(0, False), (1, False), (1, True)])
def test_skipped_rows_gradients_equal_the_oracle(cb, O, bg, z, cols, low, multi, info_only):
    """Sent lengths that leave trailing rows with an unsent own column: skipped when their
    offsets are not negative (low = 0), run otherwise; the loss over all bits or the
    information bits only.  The oracle runs every row."""
    T, n, k, e = 4, 5, (22 if bg == 1 else 10) * z, cols * z
    g = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f32")
    ref = O.Code(k, e, bg=bg, z=z)
    net = cb.LearnedNms(g, T, shared=True)
    net.set_loss_bits(info_only)
    rng = np.random.default_rng(cols)
    alpha = (0.75 + 0.05 * rng.standard_normal(net.n_weights)).astype(np.float32)
    beta = (low + 0.05 * np.abs(rng.standard_normal(net.n_weights))).astype(np.float32)
    net.set_weights(alpha, beta)
    cw = np.stack([ref.encode_full(u) for u in rng.integers(0, 2, (n, k)).astype(np.uint8)])
    llr = (2.0 * (1.0 - 2.0 * cw[:, 2 * z:2 * z + e]) + 2.0 * rng.standard_normal((n, e))).astype(np.float32)
    loss, ga, gb = net.gradients(llr, cw, multi_loss=multi)
    rloss, rpost, (rga, rgb) = ref.learned(T, True, alpha, beta, llr, cw, want_post=True, want_grad=True, multi=multi,
                                           info_only=info_only, precision="f32")
    assert np.array_equal(net.forward(llr).view(np.uint32), rpost.view(np.uint32))
    assert abs(loss - rloss) <= 1e-5 * abs(rloss)
    for got, want in ((ga, rga), (gb, rgb)):
        assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)

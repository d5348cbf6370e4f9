"""Gradients of codes with skipped rows (cbh::live_rows) after calls that left infinities in
the kept row records: base graph 2 at rate 1/2, whose last live level holds a skipped row, and
base graph 1 with 35 and with 17 live rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bg, z, cols", [(2, 52, 20), (1, 20, 55), (1, 20, 37)])
@pytest.mark.parametrize("multi", [0, 1, 2])
@pytest.mark.parametrize("info_only", [False, True])
def test_kept_records_of_skipped_rows_reach_no_gradient(cb, O, bg, z, cols, multi, info_only):
    T, n, k, e = 4, 3, (22 if bg == 1 else 10) * z, cols * z
    g = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f32")
    ref = O.Code(k, e, bg=bg, z=z)
    net = cb.LearnedNms(g, T, shared=True)
    net.set_loss_bits(info_only)
    rng = np.random.default_rng(cols + multi)
    alpha = (0.75 + 0.05 * rng.standard_normal(net.n_weights)).astype(np.float32)
    beta = (0.05 * np.abs(rng.standard_normal(net.n_weights))).astype(np.float32)
    cw = np.stack([ref.encode_full(u) for u in rng.integers(0, 2, (n, k)).astype(np.uint8)])
    llr = (2.0 * (1.0 - 2.0 * cw[:, 2 * z:2 * z + e]) + 2.0 * rng.standard_normal((n, e))).astype(np.float32)
    # negative offsets: every row runs and leaves its record, here of infinite magnitudes
    net.set_weights(alpha, -1.0 - beta)
    net.gradients(np.full_like(llr, np.nan), cw, multi_loss=multi)
    net.set_weights(alpha, beta)
    loss, ga, gb = net.gradients(llr, cw, multi_loss=multi)
    rloss, _, (rga, rgb) = ref.learned(T, True, alpha, beta, llr, cw, want_post=True, want_grad=True, multi=multi,
                                       info_only=info_only, precision="f32")
    # the bounds of tests/test_gpu_learned.py: the order of the f32 sums and CUDA's expf
    assert abs(loss - rloss) <= 1e-5 * abs(rloss)
    for got, want in ((ga, rga), (gb, rgb)):
        assert np.all(np.isfinite(got))
        assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)
    # a skipped row's edges but its own column's send zero: no gradient at all
    layer, column, _ = g.tables()[0].T
    other = (layer >= cols + 2 - k // z) & (column != k // z + layer)
    for got in (ga, gb):
        assert not np.any(got.reshape(T, -1)[:, other])

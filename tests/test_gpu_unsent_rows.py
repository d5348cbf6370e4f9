"""Decoding with the trailing rows whose own parity column is not sent skipped
(cbh::live_rows) against the oracle, which runs every row: decisions, iterations and a
posteriori LLRs bit for bit.

Sent lengths on both sides of a column's edge, from every row live to the core rows only,
both base graphs, partial warps, a scale of zero, and integer LLRs: exact zeros and ties, whose own columns are zero and whose
checks the full syndrome test must still find failing.  The learned decoder's whole
posteriors, own columns included, against its training forward (every row, every
iteration), with offsets that allow skipping and one that does not."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (base graph, Z, sent columns, sent bits more or less)
LENGTHS = [(1, 20, 66, 0), (1, 20, 65, 1), (1, 20, 44, 0), (1, 20, 44, 1), (1, 20, 44, -1), (1, 20, 26, 0), (1, 20, 24, 3),
           (2, 52, 50, 0), (2, 52, 20, 0), (2, 52, 20, -7), (2, 36, 23, 1), (2, 36, 12, 0), (2, 7, 11, 2)]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("rule, alpha", [("normalized_min_sum", 0.75), ("offset_min_sum", 0.5),
                                         ("normalized_min_sum", 0.0)])
@pytest.mark.parametrize("bg, z, cols, more", LENGTHS)
def test_skipped_rows_change_nothing(cb, O, bg, z, cols, more, rule, alpha, precision):
    k, e = (22 if bg == 1 else 10) * z, cols * z + more
    g = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision=precision, rule=rule, alpha=alpha, max_iterations=7)
    ref = O.Code(k, e, bg=bg, z=z)
    ref.set_decoder(O.RULE_OMS if rule == "offset_min_sum" else O.RULE_NMS, alpha, True, 7)
    rng = np.random.default_rng(cols * z + more)
    u = rng.integers(0, 2, (18, k)).astype(np.uint8)
    s = 1.0 - 2.0 * np.stack([ref.encode(b) for b in u])
    llr = 6.0 * s + 4.0 * rng.standard_normal(s.shape)
    llr[6:12] = np.round(llr[6:12] / 4.0)       # ties and exact zeros
    llr[12:16] = 2.0 * s[12:16] + 6.0 * rng.standard_normal((4, e))
    llr[16:] = 8.0 * s[16:]                      # the channel word of a codeword
    llr = llr.astype(g.dtype)
    bits, app, it = g.decode_full(llr)
    word = np.uint64 if precision == "f64" else np.uint32
    for f in range(len(llr)):
        rb, rit, rapp, _ = ref.decode(llr[f], precision, want_app=True)
        assert rit == it[f] and np.array_equal(rb, bits[f]), f
        assert np.array_equal(rapp.view(word), app[f].view(word)), f


@pytest.mark.parametrize("bg, z, cols", [(1, 128, 44), (2, 128, 20), (2, 52, 20), (2, 20, 13)])
@pytest.mark.parametrize("low", [0.0, -0.05])
def test_learned_posteriors_equal_the_training_forward(cb, O, bg, z, cols, low):
    k, e, T = (22 if bg == 1 else 10) * z, cols * z, 5
    g = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f32", max_iterations=T)
    net = cb.LearnedNms(g, T, shared=True)
    rng = np.random.default_rng(z + cols)
    alpha = (0.8 + 0.1 * rng.standard_normal(net.n_weights)).astype(np.float32)
    beta = (low + 0.1 * np.abs(rng.standard_normal(net.n_weights))).astype(np.float32)
    net.set_weights(alpha, beta)
    ref = O.Code(k, e, bg=bg, z=z)
    s = 1.0 - 2.0 * np.stack([ref.encode(b) for b in rng.integers(0, 2, (24, k)).astype(np.uint8)])
    llr = (3.0 * s + 3.0 * rng.standard_normal(s.shape)).astype(np.float32)
    llr[:8] = np.round(llr[:8])
    llr[20:] = (12.0 * s + 3.0 * rng.standard_normal(s.shape)).astype(np.float32)[20:]
    post, its = net.decode(llr)
    full = net.forward(llr)
    all_t = its == T
    assert np.array_equal(post[all_t].view(np.uint32), full[all_t].view(np.uint32))
    # words that stop: the training forward of as many iterations
    for t in sorted(set(its[~all_t].tolist()) - {0}):
        short = cb.LearnedNms(g, t, shared=True)
        w = net.n_weights // T * t
        short.set_weights(alpha[:w], beta[:w])
        rows = np.flatnonzero(its == t)
        assert np.array_equal(post[rows].view(np.uint32), short.forward(llr[rows]).view(np.uint32)), t

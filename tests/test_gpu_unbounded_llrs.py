"""Infinite, huge and NaN LLRs through the decoders that skip rows (cbh::live_rows).

The same channel word is decoded twice: as E sent LLRs, which leaves trailing rows with an unsent
own column, and as the whole circular buffer with LLR 0 where nothing was sent, a code whose
every row runs.  Both have the same answer bit for bit: hard decisions, iterations and
posteriors, NaNs included.  Words: erasures with certain bits, the same with errors, noisy
words with some certain, some of the largest finite magnitude, and some not numbers."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CODES = [(1, 20, 44), (1, 20, 26), (2, 52, 20), (2, 36, 12)]


def words(O, bg, z, cols, dtype):
    k, e, full = (22 if bg == 1 else 10) * z, cols * z, (66 if bg == 1 else 50) * z
    ref = O.Code(k, e, bg=bg, z=z)
    rng = np.random.default_rng(z + cols)
    cw = np.stack([ref.encode_full(u) for u in rng.integers(0, 2, (24, k)).astype(np.uint8)])
    s = 1.0 - 2.0 * cw[:, 2 * z:2 * z + e]
    y = 4.0 * s + 4.0 * rng.standard_normal(s.shape)
    erased = np.where(rng.random(s.shape) < 0.75, s * np.inf, y)
    erased[~np.isinf(erased)] = 0.0
    llr = y.copy()
    llr[0:6] = erased[0:6]
    llr[6:10] = np.where(rng.random((4, e)) < 0.03, -erased[6:10] + 0.0, erased[6:10])
    llr[10:14] = np.where(rng.random((4, e)) < 0.3, s[10:14] * np.inf, y[10:14])
    llr[14:18] = np.where(rng.random((4, e)) < 0.3, s[14:18] * float(np.finfo(dtype).max), y[14:18])
    llr[18:21] = np.where(rng.random((3, e)) < 0.05, np.nan, y[18:21])
    padded = np.zeros((len(llr), full))
    padded[:, :e] = llr
    return k, e, full, cw, llr.astype(dtype), padded.astype(dtype)


def same(a, b):
    """Equal values, zeros' signs and places of NaN."""
    return np.array_equal(a, b, equal_nan=True) and np.array_equal(np.signbit(a[a == 0]), np.signbit(b[b == 0]))


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("rule, alpha", [("normalized_min_sum", 0.75), ("offset_min_sum", 0.5),
                                         ("normalized_min_sum", 0.0), ("normalized_min_sum", 3e6)])
@pytest.mark.parametrize("bg, z, cols", CODES)
def test_unbounded_words_decode_as_with_every_row(cb, O, bg, z, cols, rule, alpha, precision):
    kw = dict(base_graph=bg, lifting_size=z, precision=precision, rule=rule, alpha=alpha, max_iterations=8)
    dtype = np.float64 if precision == "f64" else np.float32
    k, e, full, _, llr, padded = words(O, bg, z, cols, dtype)
    g, every = cb.NrLdpc(k, e, **kw), cb.NrLdpc(k, full, **kw)
    for reps in (1, 80):  # few codewords and a full device
        bits, app, its = g.decode_full(np.tile(llr, (reps, 1)))
        rbits, rapp, rits = every.decode_full(np.tile(padded, (reps, 1)))
        for f in range(len(bits)):
            assert its[f] == rits[f] and np.array_equal(bits[f], rbits[f]) and same(app[f], rapp[f]), f % len(llr)


@pytest.mark.parametrize("precision, powers", [("f64", (0, 900, 997, 1012)), ("f32", (0, 80, 97, 112))])
@pytest.mark.parametrize("bg, z, cols", CODES)
def test_large_finite_words_equal_the_oracle(cb, O, bg, z, cols, precision, powers):
    # the normalised rule commutes with a power of two while nothing overflows: magnitudes below, at
    # and beyond the bound from which every row runs, and words that pass it while decoding
    dtype = np.float64 if precision == "f64" else np.float32
    k, e = (22 if bg == 1 else 10) * z, cols * z
    g = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision=precision, max_iterations=8)
    ref = O.Code(k, e, bg=bg, z=z).set_decoder(O.RULE_NMS, 0.75, True, 8)
    rng = np.random.default_rng(cols)
    s = 1.0 - 2.0 * np.stack([ref.encode(u) for u in rng.integers(0, 2, (6, k)).astype(np.uint8)])
    llr = (3.0 * s + 4.0 * rng.standard_normal(s.shape)).astype(dtype)
    bits, app, its = g.decode_full(np.concatenate([llr * dtype(2.0) ** p for p in powers]))
    word = np.uint64 if precision == "f64" else np.uint32
    for i, p in enumerate(powers):
        for f in range(len(llr)):
            rb, rit, rapp, _ = ref.decode(llr[f] * dtype(2.0) ** p, precision, want_app=True)
            at = i * len(llr) + f
            assert np.all(np.isfinite(rapp)) and rit == its[at], (p, f)
            assert np.array_equal(rb, bits[at]) and np.array_equal(rapp.view(word), app[at].view(word)), (p, f)


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_unbounded_words_without_allocation(cb, O, precision):
    import torch

    dtype = np.float64 if precision == "f64" else np.float32
    k, e, full, _, llr, padded = words(O, 2, 36, 12, dtype)
    kw = dict(base_graph=2, lifting_size=36, precision=precision, max_iterations=8)
    g, every = cb.NrLdpc(k, e, **kw), cb.NrLdpc(k, full, **kw)
    x = torch.from_numpy(llr).cuda()
    words_out = torch.zeros(len(llr), (k + 31) // 32, dtype=torch.int32, device="cuda")
    its = torch.zeros(len(llr), dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert cb.lib().cb_decode_device_noalloc(g._h, p(x), len(llr), p(words_out), p(its), stream) == 0
    bits = np.unpackbits(words_out.cpu().numpy().view(np.uint8), axis=1, bitorder="little")[:, :k]
    rbits, _, rits = every.decode_full(padded)
    assert np.array_equal(its.cpu().numpy(), rits) and np.array_equal(bits, rbits)


@pytest.mark.parametrize("bg, z, cols", [(1, 128, 44), (2, 128, 20), (2, 52, 20)])
@pytest.mark.parametrize("own", ["plain", "large"])
def test_unbounded_words_in_the_learned_decoder(cb, O, bg, z, cols, own):
    # decoding, the training forward and the gradients; own: an own column's scale beyond what
    # keeps a skipped row's magnitudes finite
    T = 5
    k, e, full, cw, llr, padded = words(O, bg, z, cols, np.float32)
    kw = dict(base_graph=bg, lifting_size=z, precision="f32", max_iterations=T)
    nets = [cb.LearnedNms(cb.NrLdpc(k, n, **kw), T, shared=True) for n in (e, full)]
    rng = np.random.default_rng(z)
    alpha = (0.8 + 0.1 * rng.standard_normal(nets[0].n_weights)).astype(np.float32)
    beta = (0.1 * np.abs(rng.standard_normal(nets[0].n_weights))).astype(np.float32)
    if own == "large":
        alpha.reshape(T, -1)[2, -1] = 1e38
    for net in nets:
        net.set_weights(alpha, beta)
    post, its = nets[0].decode(llr)
    rpost, rits = nets[1].decode(padded)
    assert np.array_equal(its, rits)
    for f in range(len(llr)):
        assert same(post[f], rpost[f]), f
    got, want = nets[0].forward(llr), nets[1].forward(padded)
    for f in range(len(llr)):
        assert same(got[f], want[f]), f
    # gradients of a batch whose loss is finite: noisy words and, one at a time, others
    for rows in (np.r_[21:24], np.r_[14, 21:24], np.r_[10, 21:24]):
        for multi in (0, 1):
            loss, ga, gb = nets[0].gradients(llr[rows], cw[rows], multi_loss=multi)
            rloss, rga, rgb = nets[1].gradients(padded[rows], cw[rows], multi_loss=multi)
            assert np.isnan(loss) == np.isnan(rloss)
            for a, b in ((ga, rga), (gb, rgb)):
                assert np.array_equal(np.isnan(a), np.isnan(b))
                ok = np.isfinite(a) & np.isfinite(b)
                # (the order of the f32 sums, as in tests/test_gpu_learned.py)
                assert np.linalg.norm(a[ok] - b[ok]) <= 1e-4 * max(np.linalg.norm(b[ok]), 1e-30)


def test_unbounded_words_in_a_mixed_batch(cb):
    # Eb/N0 at which LLRs reach the largest floats, infinity and (0 times infinity) NaN
    items = cb.draw_mixed_batch(n=240, seed=11, zs=(16, 64, 128))
    items["ebn0_db"] = np.resize([3.0, 360.0, 372.0, 378.0, 384.0, 400.0], len(items))
    mix = cb.MixBatch(items, seed=7, name="unbounded", max_iterations=9)
    for rho in (1, 2):
        for i in range(len(mix.classes())):
            try:
                mix.set_rows_per_thread(i, rho)
            except cb.ComrsError:
                pass
        got = mix.run(0)
        llrs, infos = mix.frames(0)
        codes = {}
        for i, it in enumerate(items):
            bg, z, k = int(it["base_graph"]), int(it["lifting_size"]), int(it["k_info"])
            full = (66 if bg == 1 else 50) * z
            if (bg, z) not in codes:
                codes[bg, z] = cb.NrLdpc(k, full, base_graph=bg, lifting_size=z, precision="f32", max_iterations=9)
            word = np.zeros(full, np.float32)
            word[:len(llrs[i])] = llrs[i]
            bits, _, its = codes[bg, z].decode_full(word)
            assert its == got["iterations"][i] and int(np.sum(bits != infos[i])) == got["bit_errors"][i], (i, rho)

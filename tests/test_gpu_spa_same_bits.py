"""The generic sum-product kernels against the ones they stand in for, bit for bit, and in f32
against the oracle.

The same rows go through the other kernel when the code is given something that changes no
message: for the chained decoder (csrc/sparse_chain.cu) one more row of two variables of its
own, after which a level has two rows and a warp takes each row; for the edge-parallel one
(csrc/sparse_edges.cu) so many variables in no row that a word does not fit shared memory.
Both precisions; posteriors of the common variables and iterations are the same bits.  The
f32 posteriors of one iteration are the oracle's within what the two libraries' tanh and
atanh make of moderate LLRs.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRECISIONS = [("f64", np.uint64), ("f32", np.uint32)]


def _chain(k, m, dmin, dmax, seed):
    """An accumulator's rows: `dmin` to `dmax` - 2 information bits, the bit before and the own."""
    rng = np.random.default_rng(seed)
    rows = []
    for r in range(m):
        info = rng.choice(k, size=int(rng.integers(dmin, dmax - 1)), replace=False).tolist()
        rows.append(info + ([k + r - 1] if r else []) + [k + r])
    return k + m, rows


def _levels(n, m, dmin, dmax, seed):
    """Random rows, the first nine of them without a common variable."""
    rng = np.random.default_rng(seed)
    first = [list(range(i * dmin, (i + 1) * dmin)) for i in range(9)]
    return n, first + [sorted(rng.choice(n, size=int(rng.integers(dmin, dmax + 1)), replace=False).tolist())
                       for _ in range(m)]


CHAINS = [(6000, 700, 1, 8, 1), (40000, 333, 2, 16, 2), (300000, 260, 9, 32, 3)]
EDGES = [(60, 30, 1, 3, 1), (700, 300, 2, 9, 2), (1500, 90, 3, 40, 3), (900, 501, 2, 6, 4)]
FRAMES = [1, 5, 333]


def _same(gpu, other, llr, extra, dt):
    wide = np.concatenate([llr, np.full((len(llr), extra), 2.0)], axis=1)
    post, it = gpu.decode_llr(llr)
    rpost, rit = other.decode_llr(wide)
    assert np.array_equal(it, rit)
    assert np.array_equal(post.view(dt), np.ascontiguousarray(rpost[:, :llr.shape[1]]).view(dt))


@pytest.mark.parametrize("precision, dt", PRECISIONS)
@pytest.mark.parametrize("k, m, dmin, dmax, seed", CHAINS)
def test_chained_rows_equal_a_warp_per_row(cb, k, m, dmin, dmax, seed, precision, dt):
    n, rows = _chain(k, m, dmin, dmax, seed)
    kw = dict(max_iterations=9, precision=precision, encoder=None)
    gpu, other = cb.Ldpc(n, rows, **kw), cb.Ldpc(n + 2, rows + [[n, n + 1]], **kw)
    assert gpu.info()["max_level_rows"] == 1 and other.info()["max_level_rows"] == 2
    llr = np.random.default_rng(seed).normal(3.0, 1.8, (24, n))
    llr[:, 0] = 0.0
    llr[3, 5:9] = np.inf
    _same(gpu, other, llr, 2, dt)


@pytest.mark.parametrize("precision, dt", PRECISIONS)
@pytest.mark.parametrize("frames", FRAMES)
@pytest.mark.parametrize("n, m, dmin, dmax, seed", EDGES)
def test_edge_parallel_rows_equal_a_thread_per_row(cb, n, m, dmin, dmax, seed, frames, precision, dt):
    n, rows = _levels(n, m, dmin, dmax, seed)
    kw = dict(max_iterations=9, precision=precision, encoder=None)
    gpu, other = cb.Ldpc(n, rows, **kw), cb.Ldpc(n + 60000, rows, **kw)
    assert gpu.info()["max_level_rows"] > 8
    llr = np.random.default_rng(seed).normal(2.5, 2.0, (frames, n))
    llr[:, 0] = 0.0
    llr[0, 3] = np.inf
    _same(gpu, other, llr, 60000, dt)


@pytest.mark.parametrize("precision, dt", PRECISIONS)
@pytest.mark.parametrize("degree", [255, 256])
def test_the_longest_rows_of_an_edge_a_thread(cb, degree, precision, dt):
    # a row of 256 edges leaves the code to the kernel with several words a CTA and a thread a row
    n = 700
    rows = [list(range(degree))] + [[degree + 2 * i, degree + 2 * i + 1] for i in range(12)]
    rows += [sorted(np.random.default_rng(i).choice(n, 5, replace=False).tolist()) for i in range(60)]
    kw = dict(max_iterations=9, precision=precision, encoder=None)
    gpu, other = cb.Ldpc(n, rows, **kw), cb.Ldpc(n + 60000, rows, **kw)
    assert gpu.info()["max_level_rows"] > 8
    _same(gpu, other, np.random.default_rng(degree).normal(4.0, 2.0, (40, n)), 60000, dt)


@pytest.mark.parametrize("kind, shape", [("chain", s) for s in CHAINS] + [("edges", s) for s in EDGES])
def test_f32_agrees_with_the_oracle_after_one_iteration(cb, O, kind, shape):
    # rows of at least three edges and LLRs within +-3: a message's product of tanh values is wrong
    # by some 5 of its last bits an edge, 1e-5 for 40 edges, and stays 4e-4 below 1 (two other
    # variables of a few times +-3), where 2 atanh multiplies an error by 2 / (1 - p^2): 6e-3
    size, m, dmin, dmax, seed = shape
    n, rows = (_chain if kind == "chain" else _levels)(size, m, max(dmin, 1 if kind == "chain" else 3), max(dmax, 4), seed)
    rows = [r for r in rows if len(r) >= 3] if kind == "edges" else [[n, n + 1] + rows[0]] + rows[1:]
    n += 2
    gpu = cb.Ldpc(n, rows, max_iterations=1, precision="f32", encoder=None)
    info = gpu.info()["max_level_rows"]
    assert info == 1 if kind == "chain" else info > 8
    ref = O.Code(rows=rows, n=n)
    ref.set_decoder(O.RULE_SUM_PRODUCT, 0.0, True, 1)
    llr = np.clip(np.random.default_rng(seed).normal(1.0, 1.5, (40, n)), -3.0, 3.0).astype(np.float32)
    post_g, it_g = gpu.decode_llr(llr)
    post_o, it_o = ref.decode_llr_many(llr.astype(np.float64), "f32")
    assert np.array_equal(it_g, it_o)
    assert np.abs(post_g.astype(np.float64) - np.asarray(post_o, np.float64)).max() <= 1e-2

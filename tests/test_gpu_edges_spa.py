"""The edge-parallel layered sum-product decoder (csrc/sparse_edges.cu) against the oracle.

Rows of one to 40 edges in levels of more than eight rows, batches of one word, of fewer
words than a CTA holds and of many: iterations equal, posteriors within what the two
libraries' tanh and atanh make of 6 iterations.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, m, dmax, seed):
    rng = np.random.default_rng(seed)
    rows = [sorted(rng.choice(n, size=int(rng.integers(1, dmax + 1)), replace=False).tolist()) for _ in range(m)]
    # at least nine disjoint rows first, so that a level holds more than eight
    return [[9 * dmax + i] for i in range(9)] + rows


@pytest.mark.parametrize("frames", [1, 5, 333])
@pytest.mark.parametrize("n, m, dmax, seed", [(40, 30, 2, 1), (700, 300, 9, 2), (1500, 90, 40, 3), (900, 501, 6, 4)])
def test_edge_parallel_sum_product_agrees_with_the_oracle(cb, O, n, m, dmax, seed, frames):
    rows = _rows(n, m, dmax, seed)
    gpu = cb.Ldpc(n, rows, max_iterations=6, encoder=None)
    assert gpu.info()["max_level_rows"] > 8
    ref = O.Code(rows=rows, n=n)
    ref.set_decoder(O.RULE_SUM_PRODUCT, 0.0, True, 6)
    llr = np.random.default_rng(seed).normal(2.5, 2.0, (frames, n))
    llr[:, 0] = 0.0
    post_g, it_g = gpu.decode_llr(llr)
    post_o, it_o = ref.decode_llr_many(llr, "f64")
    assert np.array_equal(it_g, it_o)
    # the bound of the PEG codes' early words (tests/test_gpu_sparse.py)
    gap = np.abs(post_g - post_o) / np.maximum(1.0, np.abs(post_o))
    assert gap.max() <= 1e-9

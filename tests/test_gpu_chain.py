"""The chained layered decoder (csrc/sparse_chain.cu) against the oracle's sequential rows.

Irregular repeat-accumulate codes of every slot width (8, 16 and 32 edges a row), with rows
of one to 32 edges, blocks that end early on a shared information bit, and rows that share
another variable instead of the accumulator's: the min-sum rules give the oracle's
posteriors bit for bit in f64 and f32, with signed zeros and infinite LLRs among them; the
sum-product rule the oracle's outcome (its tanh and atanh are the platform libm's).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ira(k, m, dmin, dmax, seed):
    rng = np.random.default_rng(seed)
    rows = []
    for r in range(m):
        info = rng.choice(k, size=int(rng.integers(dmin, dmax - 1)), replace=False).tolist()
        if r and rng.random() < 0.02:
            # a row without the link: it shares an information bit with the row before
            prev = [v for v in rows[-1] if v < k]
            if prev and prev[0] not in info and len(info) < dmax - 1:
                rows.append(info + [prev[0], k + r])
                continue
        rows.append(info + ([k + r - 1] if r else []) + [k + r])
    return k + m, rows


def _mean_block(rows):
    """Rows per block of at most 64: the decoder takes the chained path from 16."""
    blocks, used, length = 0, set(), 64
    for r, row in enumerate(rows):
        link = rows[r - 1][-1] if r and len(row) > 1 and row[-2] == rows[r - 1][-1] else None
        if length == 64 or any(v in used and v != link for v in row):
            blocks, used, length = blocks + 1, set(), 0
        used.update(row)
        length += 1
    return len(rows) / blocks


CODES = [(6000, 700, 0, 8, 1), (40000, 333, 2, 16, 2), (300000, 260, 9, 32, 3), (400, 65, 1, 4, 4)]


@pytest.mark.parametrize("precision, dt", [("f64", np.uint64), ("f32", np.uint32)])
@pytest.mark.parametrize("rule, alpha", [("normalized_min_sum", 0.75), ("offset_min_sum", 0.3)])
@pytest.mark.parametrize("k, m, dmin, dmax, seed", CODES)
def test_min_sum_equals_the_oracle_bit_for_bit(cb, O, k, m, dmin, dmax, seed, rule, alpha, precision, dt):
    n, rows = _ira(k, m, dmin, dmax, seed)
    gpu = cb.Ldpc(n, rows, rule=rule, alpha=alpha, max_iterations=9, precision=precision, encoder=None)
    assert gpu.info()["max_level_rows"] == 1 and _mean_block(rows) >= 16
    ref = O.Code(rows=rows, n=n)
    ref.set_decoder({"normalized_min_sum": O.RULE_NMS, "offset_min_sum": O.RULE_OMS}[rule], alpha, True, 9)
    rng = np.random.default_rng(seed)
    llr = rng.normal(3.0, 1.6, (24, n))
    llr[:, :3] = 0.0
    llr[:8, 3:7] = -0.0
    llr[8:12, 7] = np.inf
    post_g, it_g = gpu.decode_llr(llr)
    post_o, it_o = ref.decode_llr_many(llr, precision)
    assert np.array_equal(it_g, it_o)
    assert np.array_equal(post_g.view(dt), post_o.view(dt))


@pytest.mark.parametrize("k, m, dmin, dmax, seed", CODES)
def test_sum_product_agrees_with_the_oracle(cb, O, k, m, dmin, dmax, seed):
    n, rows = _ira(k, m, dmin, dmax, seed)
    gpu = cb.Ldpc(n, rows, max_iterations=9, encoder=None)
    ref = O.Code(rows=rows, n=n)
    ref.set_decoder(O.RULE_SUM_PRODUCT, 0.0, True, 9)
    llr = np.random.default_rng(seed).normal(3.0, 1.6, (24, n))
    post_g, it_g = gpu.decode_llr(llr)
    post_o, it_o = ref.decode_llr_many(llr, "f64")
    assert np.array_equal(it_g, it_o)
    # the two libm's last bits through 9 iterations (the bound of the PEG codes' test)
    assert np.abs(post_g - post_o).max() <= 1e-9 * max(1.0, np.abs(post_o).max())

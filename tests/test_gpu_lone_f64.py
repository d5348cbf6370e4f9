"""f64 decoding of a few codewords (rows with the base graph at compile time) against the
full device's build on the same frames: the same records, both base graphs, both rules,
whole and partial warps, one and several warps, the largest and the smallest lifting."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule, alpha", [("normalized_min_sum", 0.75), ("offset_min_sum", 0.5)])
@pytest.mark.parametrize("bg, z, n", [(1, 2, 6000), (1, 36, 2500), (1, 144, 700), (1, 384, 200), (2, 2, 6000),
                                      (2, 52, 2500), (2, 64, 2500), (2, 384, 200)])
def test_lone_frames_equal_the_full_device(cb, bg, z, n, rule, alpha):
    k = (22 if bg == 1 else 10) * z
    for e in (2 * k, 3 * k - 1):
        g = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f64", rule=rule, alpha=alpha, max_iterations=12)
        full = g.run_frames(3, "lone", 0, 0, n, 1.2, 4)
        assert np.array_equal(g.run_frames(3, "lone", 0, 0, 40, 1.2, 4), full[:40])
        assert np.array_equal(g.run_frames(3, "lone", 0, 50, 1, 1.2, 4), full[50:51])

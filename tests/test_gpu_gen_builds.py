"""The f64 generator's builds (gen.cu): frames of the exact 256-point demapper generated in one
call of several rounds and in calls of a few frames are the same, at frames of more and of
fewer symbols than the line between them."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z, cols", [(52, 20), (50, 20)])
def test_the_builds_generate_the_same_frames(cb, z, cols):
    import torch

    n = 12 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    g = cb.NrLdpc(10 * z, cols * z, base_graph=2, lifting_size=52, precision="f64", demapper="exact")
    llr, info = g.generate_frames(5, "builds", 0, 0, n, 10.0, 256)
    for first in (0, n // 2, n - 40):
        l, i = g.generate_frames(5, "builds", 0, first, 40, 10.0, 256)
        assert np.array_equal(l.view(np.uint64), llr[first:first + 40].view(np.uint64))
        assert np.array_equal(i, info[first:first + 40])

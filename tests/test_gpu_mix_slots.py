"""Mixed batches: the slots a CTA opens and the row code they run do not change a record.

Small and larger batches (one and several slots of a class per CTA), liftings on both
sides of 128 threads per slot (straight-line rows from there) and ones that leave part of a
slot's last warp idle, both base graphs: every record equals the single-code path's."""

import numpy as np
import pytest

from test_gpu_mix import NAME, single_code_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zs, n", [((16, 24, 32), 400), ((30, 36, 60, 64), 60), ((96, 104, 128, 112), 60),
                                   ((120, 176, 208, 256), 60), ((288, 320, 352, 384), 60), ((128,), 1), ((384,), 700)])
def test_mixed_records_equal_the_single_code_path(cb, zs, n):
    items = cb.draw_mixed_batch(n=n, seed=n + zs[0], zs=zs)
    got = cb.MixBatch(items, seed=7, name=NAME, max_iterations=25).run(0)
    assert np.array_equal(got, single_code_records(cb, items, 0, n))

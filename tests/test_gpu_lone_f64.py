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


def test_no_alloc_calls_after_the_first_map_no_kernel(cb):
    # One call on a small code loads all of the f64 decoder's builds: calls on the other base
    # graph, with few and with many codewords, leave the free device memory as it was, and
    # decide as the allocating decoder.
    import ctypes as C

    import torch

    def setup(bg, z, n):
        k, e = (22 if bg == 1 else 10) * z, (44 if bg == 1 else 20) * z
        code = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f64")
        gen = cb.NrLdpc(k, e, base_graph=bg, lifting_size=z, precision="f64")
        llr = torch.from_numpy(gen.generate_frames(7, "no_alloc_f64", 0, 0, n, 1.0, 4)[0]).cuda()
        out = [torch.full((n, (k + 31) // 32), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
        its = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
        return code, gen, llr, out, its

    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    L, ptr = cb.lib(), (lambda t: C.c_void_p(t.data_ptr()))
    cases = [setup(2, 52, 4), setup(1, 36, 4), setup(1, 36, 2500), setup(2, 52, 2500)]
    torch.cuda.synchronize()
    for i, (code, _, llr, out, its) in enumerate(cases):
        free = torch.cuda.mem_get_info()[0]
        assert L.cb_decode_device_noalloc(code._h, ptr(llr), len(llr), ptr(out[0]), ptr(its[0]), stream) == 0
        torch.cuda.synchronize()
        assert i == 0 or torch.cuda.mem_get_info()[0] == free, i
    for code, gen, llr, out, its in cases:
        assert L.cb_decode_device(gen._h, ptr(llr), len(llr), ptr(out[1]), None, ptr(its[1]), stream) == 0
        torch.cuda.synchronize()
        assert torch.equal(out[0], out[1]) and torch.equal(its[0], its[1])


@pytest.mark.parametrize("bg, z, per_sm", [(1, 32, (3, 4)), (1, 64, (3, 4)), (1, 96, (2, 3)), (1, 120, (3, 4)),
                                           (2, 20, (15, 16)), (2, 52, (7, 8)), (2, 128, (3, 4)), (2, 208, (2, 3))])
def test_the_builds_agree_at_the_line_between_them(cb, bg, z, per_sm):
    # codeword counts on both sides of the CTAs per SM at which the build changes
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    k, cols = (22 if bg == 1 else 10) * z, 66 if bg == 1 else 50
    g = cb.NrLdpc(k, cols * z, base_graph=bg, lifting_size=z, precision="f64", max_iterations=6)
    runs = [g.run_frames(3, "line", 0, 0, p * sms + d, 0.0, 4) for p in per_sm for d in (0, 1)]
    for r in runs[:-1]:
        assert np.array_equal(r, runs[-1][:len(r)])

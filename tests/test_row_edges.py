"""Rows at every alignment: what the chunk kernel's copies read, and the logits at the edges of a buffer."""
import ctypes as C

import pytest
import torch

from colinfer_b200 import _lib
from colinfer_b200 import workloads as wl


@pytest.mark.parametrize("elt,dtype", [(4, _lib.F32), (2, _lib.BF16)])
def test_copies_stay_inside_the_buffer(built_lib, elt, dtype):
    begin, end = C.c_int64(), C.c_int64()
    for addr in range(1 << 20, (1 << 20) + 32, elt):
        for V in (1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 511, 512, 513, 100_003):
            for rows in (1, 2, 3, 150):
                for row in {0, 1, 2, 3, rows // 2, rows - 4, rows - 3, rows - 2, rows - 1} & set(range(rows)):
                    assert _lib.lib().colinfer_sample_copy_range(addr, dtype, rows, V, row, C.byref(begin), C.byref(end)) == 0
                    b, e, lo, hi = begin.value, end.value, row * V * elt, (row + 1) * V * elt
                    assert 0 <= b <= e <= rows * V * elt, (addr, V, rows, row, b, e)
                    if b < e:
                        assert (addr + b) % 16 == 0 and (addr + e) % 16 == 0
                        assert b < lo + 16 and e > hi - 16               # at most part of a unit is left to ordinary loads


# the last chunk of the buffer's last row holds less than a unit, and is beyond those that a warp asks for before its first one is read:
# a CTA per row (33 chunks, 12 warps), clusters of two and of four (193 and 321 chunks, 32 and 64 warps)
SHORT_TAILS = [(149, 16_385), (57, 98_305), (33, 163_841)]


@pytest.mark.parametrize("rows,V", SHORT_TAILS)
@pytest.mark.parametrize("elt,dtype", [(4, _lib.F32), (2, _lib.BF16)])
def test_nothing_is_copied_of_a_chunk_without_a_whole_unit(built_lib, rows, V, elt, dtype):
    begin, end = C.c_int64(), C.c_int64()
    assert _lib.lib().colinfer_sample_copy_range(1 << 20, dtype, rows, V, rows - 1, C.byref(begin), C.byref(end)) == 0
    lo, hi = (rows - 1) * V * elt // 16 * 16, rows * V * elt
    assert end.value < hi and end.value == lo + (hi - lo - 1) // (512 * elt) * (512 * elt)


# a CTA per row and a cluster per row; rows of less than a unit, around a chunk of 512, and an odd one of many chunks
@pytest.mark.gpu
@pytest.mark.parametrize("rows,V", [(150, 1), (151, 3), (150, 5), (149, 511), (150, 513), (301, 4097), (40, 98_307)] + SHORT_TAILS)
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rows_of_a_buffer_at_any_alignment_draw_the_same_tokens(rows, V, dtype):
    """The first and last logits of the buffer decide (they are among the largest of their rows), and infinities surround it."""
    from colinfer_b200.spec.accept import draw
    dt = getattr(torch, dtype)
    g = torch.Generator().manual_seed(rows + V)
    x = torch.randn(rows, V, generator=g)
    x[:, :3] += 6.0
    x[:, -3:] += 6.0
    x = x.to(dt)
    params = wl._params(rows, V, torch.where(torch.arange(rows) % 5 == 4, 0.0, 0.9), torch.tensor([V, 2, 50, V, V])[torch.arange(rows) % 5].clamp_max(V),
                        torch.where(torch.arange(rows) % 3 == 0, 0.7, 1.0), torch.zeros(rows))
    sp = wl.sampler_params(params, V, "cuda")
    u = wl.open_unit(g, rows, 1).cuda()
    want, st = draw(x.cuda().view(rows, 1, V), sp, None, u=u, status=True)
    unit = 16 // x.element_size()
    for off in range(unit):
        buf = torch.full((rows * V + 2 * unit,), float("inf"), dtype=dt, device="cuda")
        view = buf[off:off + rows * V].view(rows, 1, V)
        view.copy_(x.view(rows, 1, V))
        got, st2 = draw(view, sp, None, u=u, status=True)
        assert torch.equal(got, want) and torch.equal(st2, st), off

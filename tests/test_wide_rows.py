"""Rows that are cut by more than a short list -- a top_k above a hundred, a top_p whose nucleus has thousands of logits -- where the
estimates that steer the chunk and the streaming kernel can go wrong: against the CPU oracle."""
import numpy as np
import pytest
import torch

from colinfer_b200 import _lib
from colinfer_b200 import workloads as wl
from oracle import oracle as O

from test_gpu_parity import check_tokens, mods, np_params

pytestmark = pytest.mark.gpu


def _draw(logits, params, u, flags, what, few):
    m = mods()
    V = logits.size(-1)
    out, st = m["draw"](logits.cuda(), wl.sampler_params(params, V, "cuda"), None, u=u.cuda(), status=True, flags=flags)
    want, info = O.draw(logits[few].float().numpy(), {n: v[few] for n, v in np_params(params).items()}, None, u=u[few].numpy())
    check_tokens(out.cpu().numpy()[few], want, info, what)
    return st


def _slow(st):
    return int((st & _lib.ROW_SELECT_SLOW).ne(0).sum())


# a cluster per row, the streaming kernel, a CTA per row, more rows than the SMs hold CTAs, one CTA per SM
@pytest.mark.parametrize("rows,V,hist", [(60, 151_936, 0), (100, 151_936, 0), (150, 151_936, 0), (300, 100_003, 0), (150, 216_064, 64)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_ordinary_rows_take_no_exact_select(rows, V, hist, dtype):
    """Whatever the estimates say the tokens are the oracle's: that they hold shows in the status.  N(0, 2^2), filters as they are used."""
    m = mods()
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = (torch.randn(rows, 1, V, generator=g, device="cuda") * 2).to(getattr(torch, dtype))
    n = torch.arange(rows)
    k, p = torch.tensor([V, 20, 100, 500, 1000, 1000])[n % 6], torch.tensor([0.8, 0.95, 0.9, 1.0, 0.98])[n % 5]
    sp = wl.sampler_params(wl._params(rows, V, torch.tensor([0.6, 0.8, 1.0])[n % 3], k, p, torch.where(n % 4 == 3, 0.01, 0.0)), V, "cuda")
    if hist:
        sp.set_history(torch.randint(0, V, (rows, hist), generator=g, device="cuda", dtype=torch.int32), torch.full((rows,), hist, dtype=torch.int32, device="cuda"))
        sp._ensure_penalties()
        sp.repetition_penalty.fill_(1.2)
    _, st = m["draw"](x, sp, None, u=wl.open_unit(torch.Generator().manual_seed(1), rows, 1).cuda(), status=True, flags=_lib.KERNEL_AUTO)
    print(f"{_slow(st)} of {rows} rows slow")
    assert _slow(st) <= rows // 30


# a cluster per row, a CTA per row, more rows than the SMs hold CTAs
@pytest.mark.parametrize("rows,V", [(36, 40_003), (150, 40_003), (300, 33_000)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_every_size_of_a_top_k(rows, V, dtype):
    """From the shortest that is not finished by one warp over what one pass can list to what takes a histogram and the exact select
    over the keys, with and without a top_p and a min_p that cuts above and below the k-th largest."""
    g = torch.Generator().manual_seed(rows)
    x = (torch.randn(rows, 1, V, generator=g) * 2).to(getattr(torch, dtype))
    n = torch.arange(rows)
    k = torch.tensor([101, 127, 500, 1000, 1300, 2500, V - 1])[n % 7]
    p = torch.where(n % 2 == 0, 1.0, 0.9)
    mp = torch.tensor([0.0, 0.005, 0.2])[n % 3]
    params = wl._params(rows, V, torch.where(n % 5 == 0, 0.6, 1.0), k, p, mp)
    _draw(x, params, wl.open_unit(g, rows, 1), _lib.KERNEL_AUTO, f"top_k, {rows} x {V} {dtype}", list(range(14)) + [rows - 1])


@pytest.mark.parametrize("rows,V", [(150, 40_003), (300, 33_000), (150, 151_936)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_top_k_that_removes_nothing_leaves_the_band_in_its_place(rows, V, dtype):
    """A top_k beyond what one pass lists, of which fewer logits have any mass, and a top_p: the row is counted in full, cut by its mass
    alone, and takes no exact select."""
    g = torch.Generator().manual_seed(rows + 7)
    x = (torch.randn(rows, 1, V, generator=g) * 2).to(getattr(torch, dtype))
    n = torch.arange(rows)
    T = (0.26 if V < 50_000 else 0.2) - 0.02 * (n % 3)
    params = wl._params(rows, V, T, torch.full((rows,), 10_000), torch.tensor([0.95, 0.8, 0.99])[n // 3 % 3], torch.zeros(rows))
    st = _draw(x, params, wl.open_unit(g, rows, 1), _lib.KERNEL_AUTO, f"top_k 10,000, {rows} x {V} {dtype}", list(range(9)) + [rows - 1])
    assert _slow(st) == 0


@pytest.mark.parametrize("rows", [36, 150])
def test_rows_that_mislead_the_sample(rows):
    """The sample is the first chunks of the warps and a quarter of all others; the mass that the first pass sums is relative to the
    sample's maximum.  Logits that rise or fall along the row, a period of the sample's stride, a few tokens that hold the mass and
    lie outside the sample, one so far above it that the sum overflows, rows of two values, rows mostly -inf."""
    V = 40_003
    g = torch.Generator().manual_seed(rows + 1)
    x = torch.randn(rows, 1, V, generator=g) * 2
    t = torch.arange(V)
    for r in range(rows):
        kind = r % 8
        if kind == 1:
            x[r, 0] = x[r, 0] * 0.1 + t * (8.0 / V)
        elif kind == 2:
            x[r, 0] = x[r, 0] * 0.1 - t * (8.0 / V)
        elif kind == 3:
            x[r, 0] += 3.0 * ((t // 128) % 4 == (t // 512) % 4)
        elif kind == 4:
            x[r, 0, 39_000:39_040] += 9.0
        elif kind == 5:
            x[r, 0, 38_999] = 300.0
        elif kind == 6:
            x[r, 0] = torch.where(torch.rand(V, generator=g) < 0.3, 1.0, 0.0)
        elif kind == 7:
            x[r, 0, torch.rand(V, generator=g) < 0.99] = float("-inf")
    n = torch.arange(rows)
    params = wl._params(rows, V, torch.tensor([0.5, 0.8, 1.2])[n // 8 % 3], torch.full((rows,), V), torch.tensor([0.8, 0.95, 0.999])[n % 3], torch.zeros(rows))
    _draw(x, params, wl.open_unit(g, rows, 1), _lib.KERNEL_AUTO, f"misleading rows, {rows}", list(range(24)) + [rows - 1])


@pytest.mark.parametrize("rows", [297, 298, 432, 444, 445, 593])
def test_launches_whose_last_turn_is_half_full(rows):
    """Around the row counts (half a turn of two CTAs on 148 SMs) from and up to which the second CTA of an SM starts later."""
    V = 3000
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, 1, V, generator=g) * 2
    n = torch.arange(rows)
    params = wl._params(rows, V, torch.where(n % 3 == 2, 0.0, 0.9), torch.tensor([V, V, 40])[n % 3], 0.95, 0.0)
    _draw(x, params, wl.open_unit(g, rows, 1), _lib.KERNEL_AUTO, f"{rows} rows", list(range(0, rows, 37)) + [rows - 1])


# rows of 151,936 logits: the second CTA is late by 38,000 cycles (fp32) or 19,000; more rows than are dealt by cost (16,384)
@pytest.mark.parametrize("rows,V,dtype", [(298, 151_936, "float32"), (432, 151_936, "bfloat16"), (16_385, 700, "float32"), (16_385, 700, "bfloat16")])
def test_late_starts_of_long_rows_and_of_rows_that_are_not_dealt(rows, V, dtype):
    g = torch.Generator().manual_seed(rows)
    x = (torch.randn(rows, 1, V, generator=g) * 2).to(getattr(torch, dtype))
    n = torch.arange(rows)
    params = wl._params(rows, V, torch.where(n % 7 == 6, 0.0, 0.9), torch.tensor([V, V, 40])[n % 3], 0.95, 0.0)
    few = sorted({0, 1, 2, 147, 148, 149, 150, 295, 296, 297, rows // 2, rows - 2, rows - 1})
    _draw(x, params, wl.open_unit(g, rows, 1), _lib.KERNEL_AUTO, f"{rows} x {V} {dtype}", few)


@pytest.mark.parametrize("dtype,levels,hist", [("bfloat16", 0, 0), ("bfloat16", 4, 0), ("float32", 8, 0), ("float32", 0, 0), ("bfloat16", 4, 200)])
def test_the_streaming_kernels_band_of_thousands_of_equal_logits(dtype, levels, hist):
    """Bands that overflow the lists: the pivot by narrowing the band's keys, or all keys where the band is off it as well."""
    rows, V = 24, 61_440
    m = mods()
    g = torch.Generator().manual_seed(levels + hist)
    x = torch.randn(rows, 1, V, generator=g)
    if levels:
        x = torch.round(x * levels) / levels
    x = x.to(getattr(torch, dtype))
    n = torch.arange(rows)
    params = wl._params(rows, V, torch.where(n % 2 == 0, 0.9, 1.3), torch.full((rows,), V), torch.tensor([0.8, 0.95, 0.999, 0.99999])[n % 4], torch.zeros(rows))
    u = wl.open_unit(g, rows, 1)
    if not hist:
        st = _draw(x, params, u, _lib.KERNEL_STREAM, f"equal logits, {dtype} {levels}", list(range(12)))
        off = _draw(x, params, u, _lib.KERNEL_STREAM | _lib.TEST_MISS_BAND, f"and a band off the pivot, {dtype} {levels}", list(range(12)))
        assert not levels or _slow(st) > 0                           # (the bands did overflow, the hook did move them)
        assert _slow(off) > _slow(st) or _slow(st) == rows
        return
    sp = wl.sampler_params(params, V, "cuda")
    h = torch.randint(0, V, (rows, hist), generator=g, dtype=torch.int32)
    sp.set_history(h.cuda(), torch.full((rows,), hist, dtype=torch.int32, device="cuda"))
    sp._ensure_penalties()
    sp.repetition_penalty.fill_(1.2), sp.presence_penalty.fill_(0.3), sp.frequency_penalty.fill_(0.1)
    out = m["draw"](x.cuda(), sp, None, u=u.cuda(), flags=_lib.KERNEL_STREAM).cpu().numpy()
    few, one = np.arange(12), np.ones(12, np.float32)
    pr = {k: v[few] for k, v in np_params(params).items()}
    pr.update(repetition_penalty=np.float32(1.2) * one, presence_penalty=np.float32(0.3) * one, frequency_penalty=np.float32(0.1) * one)
    want, info = O.draw(x[few].float().numpy(), pr, None, history=h[few].numpy(), hist_len=np.full(12, hist), u=u[few].numpy())
    check_tokens(out[few], want, info, "equal logits with penalties")

"""What the sampler's kernels do when an estimate is off, a list too short or a copy never arrives: the exact selects behind the
estimates, and the end of the bounded waits.  (The streaming kernel's: test_gpu_parity.py.)"""
import math

import numpy as np
import pytest
import torch

from colinfer_b200 import _lib
from colinfer_b200 import workloads as wl
from oracle import oracle as O

from test_gpu_parity import check_tokens, mods, np_params

pytestmark = pytest.mark.gpu
# rows, vocabulary, flags: the cluster-resident kernel; the chunk kernel with a CTA per row (more rows than SMs; more than they hold
# CTAs) and with a cluster of four or two per row (where no cluster of two holds the row).  Odd vocabularies: only the chunk kernel
# takes rows at any alignment through bulk copies.
FORMS = {"cluster8": (6, 33_001, _lib.KERNEL_CLUSTER[8]), "cluster4": (6, 33_001, _lib.KERNEL_CLUSTER[4]),
         "chunk": (150, 33_001, _lib.KERNEL_AUTO), "chunk, queue": (320, 33_001, _lib.KERNEL_AUTO),
         "chunk, two": (60, 98_305, _lib.KERNEL_AUTO), "chunk, four": (34, 98_307, _lib.KERNEL_AUTO)}


def _flat(form, dtype, seed, top_p=0.9):
    rows, V, flags = FORMS[form]
    g = torch.Generator().manual_seed(seed)
    logits = torch.randn(rows, 1, V, generator=g).to(dtype)
    params = wl._params(rows, V, torch.full((rows,), 0.8), torch.full((rows,), V), torch.full((rows,), top_p), torch.zeros(rows))
    return logits, params, wl.open_unit(g, rows, 1), flags


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("form", list(FORMS))
def test_a_band_off_the_pivot_is_found_out(form, dtype):
    """Rows whose nucleus holds thousands of logits, the band misplaced by the test flag (above the pivot on odd rows, below it on
    even ones): the same tokens, and the rows say that the exact select ran."""
    m = mods()
    logits, params, u, flags = _flat(form, getattr(torch, dtype), 31)
    sp = wl.sampler_params(params, logits.size(-1), "cuda")
    x, uc = logits.cuda(), u.cuda()
    good, st = m["draw"](x, sp, None, u=uc, status=True, flags=flags)
    got, st2 = m["draw"](x, sp, None, u=uc, status=True, flags=flags | _lib.TEST_MISS_BAND)
    assert torch.equal(got, good)
    assert (st2 & _lib.ROW_SELECT_SLOW).ne(0).all()
    if dtype == "float32":                                       # (bf16: a band may hold more equal logits than the lists)
        assert int((st & _lib.ROW_SELECT_SLOW).ne(0).sum()) <= len(st) // 50
    few = [0, 1, len(good) - 1]
    want, info = O.draw(logits[few].float().numpy(), {n: v[few] for n, v in np_params(params).items()}, None, u=u[few].numpy())
    check_tokens(got.cpu().numpy()[few], want, info, f"band off, {form} {dtype}")


@pytest.mark.parametrize("rows,V", [(3, 151_936), (24, 151_936), (24, 65_536), (5, 32_000)])
def test_a_top_k_of_a_thousand_fits_the_lists_of_every_cluster(rows, V):
    """Clusters of eight, four, two and one: a cluster's lists hold the same number of logits whatever its size, so that a top_k of
    a thousand needs no exact select.  (In 64 warps of 24 entries each a thousand evenly spread logits overflowed one: the launch
    of 24 rows took 99 us instead of 43.)"""
    m = mods()
    g = torch.Generator().manual_seed(rows + V)
    x = (torch.randn(rows, 1, V, generator=g) * 2).cuda()
    params = wl._params(rows, V, torch.ones(rows), torch.full((rows,), 1000), torch.full((rows,), 0.98), torch.full((rows,), 0.01))
    sp = wl.sampler_params(params, V, "cuda")
    u = wl.open_unit(g, rows, 1)
    got, st = m["draw"](x, sp, None, u=u.cuda(), status=True, flags=_lib.KERNEL_AUTO)
    assert int(st.abs().sum()) == 0
    want, info = O.draw(x[:2].cpu().numpy(), {n: v[:2] for n, v in np_params(params).items()}, None, u=u[:2].numpy())
    check_tokens(got.cpu().numpy()[:2], want, info, f"top_k 1000, {rows} x {V}")


@pytest.mark.parametrize("form", ["chunk", "chunk, queue", "chunk, two", "chunk, four"])
def test_copies_that_never_arrive_end_the_launch(form):
    """With the test flag no copy is asked for: every wait runs out (a fifth of a second, once per CTA), every row reports it, the
    kernel returns and the next launch is clean."""
    m = mods()
    logits, params, u, flags = _flat(form, torch.float32, 32)
    sp = wl.sampler_params(params, logits.size(-1), "cuda")
    x, uc = logits.cuda(), u.cuda()
    good, st = m["draw"](x, sp, None, u=uc, status=True, flags=flags)
    _, st2 = m["draw"](x, sp, None, u=uc, status=True, flags=flags | _lib.TEST_DROP_COPY)
    torch.cuda.synchronize()
    assert (st2 & _lib.ROW_TIMEOUT).ne(0).all()
    again, st3 = m["draw"](x, sp, None, u=uc, status=True, flags=flags)
    assert torch.equal(again, good) and torch.equal(st3, st) and int((st & _lib.ROW_TIMEOUT).sum()) == 0


@pytest.mark.parametrize("rows,V,dtype", [(150, 151_936, "float32"), (444, 60_000, "float32"), (60, 151_936, "bfloat16"), (300, 151_937, "bfloat16")])
def test_a_lost_copy_leaves_none_under_way(rows, V, dtype):
    """With the test flag every other warp's copies never come: the others go on reading theirs to the end of the row, and of the rows
    after it, so that none lands in shared memory that is another CTA's by then: launches on its heels, of rows of several passes, are
    as without it."""
    m = mods()
    g = torch.Generator().manual_seed(rows)
    x = (torch.randn(rows, 1, V, generator=g) * 2).to(getattr(torch, dtype)).cuda()
    n = torch.arange(rows)
    params = wl._params(rows, V, 0.8, torch.tensor([V, 40, 1000])[n % 3], torch.tensor([0.95, 1.0])[n % 2], 0.0)
    sp = wl.sampler_params(params, V, "cuda")
    u = wl.open_unit(g, rows, 1).cuda()
    good, st = m["draw"](x, sp, None, u=u, status=True, flags=_lib.KERNEL_AUTO)
    for _ in range(2):
        _, lost = m["draw"](x, sp, None, u=u, status=True, flags=_lib.KERNEL_AUTO | _lib.TEST_DROP_COPY)
        runs = [m["draw"](x, sp, None, u=u, status=True, flags=_lib.KERNEL_AUTO) for _ in range(3)]
        assert (lost & _lib.ROW_TIMEOUT).ne(0).all()
        for got, st2 in runs:
            assert torch.equal(got, good) and torch.equal(st2, st)


@pytest.mark.parametrize("rows,V", [(34, 98_320), (60, 98_307), (150, 20_000), (301, 4_099)])
def test_random_rows_of_every_form_of_the_chunk_kernel(rows, V):
    """Random value shapes (ties, runs of -inf, dominant tokens, flat and wide rows), filters, masks and histories through the chunk
    kernel with clusters of four and of two, with a CTA per row and with rows off the queue."""
    m = mods()
    for case in range(6):
        rng = np.random.default_rng(rows * 100 + case)
        g = torch.Generator().manual_seed(rows * 100 + case)
        dtype = torch.bfloat16 if case % 3 == 2 else torch.float32
        x = torch.randn(rows, 1, V, generator=g) * torch.tensor(rng.choice([1e-3, 1.0, 2.0, 30.0], size=(rows, 1, 1)), dtype=torch.float32)
        x[::4] = (x[::4] * 3).round() * 0.5
        x[1::4, :, int(rng.integers(0, V))] += 15.0
        x[2::8][torch.rand(x[2::8].shape, generator=g) < 0.5] = -math.inf
        x = x.to(dtype)
        params = wl._params(rows, V, torch.tensor(rng.choice([0.0, 0.3, 1.0, 1.5], size=rows), dtype=torch.float32),
                            torch.tensor(rng.choice([0, 1, 20, 100, 1000, V], size=rows)),
                            torch.tensor(rng.choice([1.0, 0.99, 0.9, 0.5, 1e-4], size=rows), dtype=torch.float32),
                            torch.tensor(rng.choice([0.0, 0.0, 0.01, 0.2], size=rows)))
        u = wl.open_unit(g, rows, 1)
        words = history = None
        if case % 2:
            allowed = torch.rand(rows, 1, V, generator=g) < 0.3
            allowed[..., V // 3] = True
            words = wl.pack_mask(allowed)
        sp = wl.sampler_params(params, V, "cuda")
        few = np.unique(rng.integers(0, rows, 12))
        pr = {n: v[few] for n, v in np_params(params).items()}
        if case >= 3:
            history = torch.randint(-1, V + 1, (rows, 700), generator=g, dtype=torch.int32)
            sp.set_history(history.cuda(), torch.full((rows,), 700, dtype=torch.int32, device="cuda"))
            sp._ensure_penalties()
            sp.repetition_penalty.fill_(1.3), sp.presence_penalty.fill_(0.4), sp.frequency_penalty.fill_(0.2)
            one = np.ones(len(few), np.float32)
            pr.update(repetition_penalty=np.float32(1.3) * one, presence_penalty=np.float32(0.4) * one, frequency_penalty=np.float32(0.2) * one)
        out = m["draw"](x.cuda(), sp, None, u=u.cuda(), mask=None if words is None else words.cuda(), flags=_lib.KERNEL_AUTO).cpu().numpy()
        want, info = O.draw(x[few].float().numpy(), pr, None, mask=None if words is None else words[few].numpy(),
                            history=None if history is None else history[few].numpy(), hist_len=None if history is None else np.full(len(few), 700),
                            u=u[few].numpy())
        check_tokens(out[few], want, info, f"random, {rows} x {V}, case {case}")

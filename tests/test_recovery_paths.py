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
FORMS = {"cluster8": (6, 33_001, _lib.KERNEL_CLUSTER[8]), "cluster4": (6, 33_001, _lib.KERNEL_CLUSTER[4])}


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
    assert int((st & _lib.ROW_SELECT_SLOW).ne(0).sum()) <= (0 if dtype == "float32" else len(st))
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

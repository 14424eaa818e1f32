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

"""bf16 rows away from zero, where thousands of logits share every value: the value at which a top-p cuts them has to be the oracle's,
also where the estimated band holds one value only, or misses the pivot by one."""
import numpy as np
import pytest
import torch

from colinfer_b200 import _lib
from colinfer_b200 import workloads as wl

from _oracle_pool import oracle_draw_rows
from test_gpu_parity import check_tokens, mods, np_params

pytestmark = pytest.mark.gpu
# N(mean, std^2), or three equal groups; 100 rows each, of which one to seven were cut a value too high by a band taken on trust, in one form or more
SHAPES = {"16": (16.0, 1.0), "-16": (-16.0, 1.0), "30": (30.0, 1.5), "-20": (-20.0, 2.0), "groups": None}
# the streaming kernel; the chunk kernel with a CTA per row, with a cluster per row, with rows off the queue
FORMS = {"stream": (25, _lib.KERNEL_STREAM), "chunk": (150, _lib.KERNEL_AUTO), "chunk, cluster": (36, _lib.KERNEL_AUTO), "chunk, queue": (300, _lib.KERNEL_AUTO)}
SEEDS = {"16": 5, "-16": 3, "30": 2, "-20": 2, "groups": 3}
_pool = {}


def make(shape, seed):
    """(logits, params, u) of 100 rows."""
    n = 100
    g = torch.Generator().manual_seed(seed)
    T = 0.5 + 0.7 * torch.rand(n, generator=g)
    if SHAPES[shape]:
        V, (mean, std) = 151_936, SHAPES[shape]
        x = (torch.randn(n, 1, V, generator=g) * std + mean).bfloat16()
        top_p = 0.8 + 0.19 * torch.rand(n, generator=g)
    else:
        # three equal groups: the mass of the largest, or of the two largest, is just below top_p, or just above it
        V = 61_440
        x = torch.tensor([20.25, 20.0, 19.75])[torch.stack([torch.randperm(V, generator=g) for _ in range(n)]) * 3 // V][:, None].bfloat16()
        w = torch.exp(torch.tensor([[0.0, -0.25, -0.5]]).double() / T[:, None].double())
        share = (w.cumsum(1) / w.sum(1, keepdim=True))[torch.arange(n), (torch.arange(n) % 3 > 0).long()]
        top_p = (share + 10.0 ** (-5 + 1.5 * torch.rand(n, generator=g)) * torch.where(torch.arange(n) % 4 == 3, -1.0, 1.0)).float()
    return x, wl._params(n, V, T, torch.full((n,), V), top_p, torch.zeros(n)), wl.open_unit(g, n, 1)


def _rows(shape):
    """The rows with the oracle's tokens and margins, worked out once."""
    if shape not in _pool:
        x, params, u = make(shape, SEEDS[shape])
        _pool[shape] = (x, params, u, *oracle_draw_rows(x.float().numpy(), np_params(params), None, u=u.numpy()))
    return _pool[shape]


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("shape", list(SHAPES))
def test_coarse_rows_are_cut_at_the_oracles_value(shape, form):
    m = mods()
    rows, flags = FORMS[form]
    x, params, u, want, info = _rows(shape)
    for lo in range(0, 100, rows):
        at = (torch.arange(rows) + lo) % 100
        sp = wl.sampler_params({k: v[at] for k, v in params.items()}, x.size(-1), "cuda")
        got = m["draw"](x[at].cuda(), sp, None, u=u[at].cuda(), flags=flags).cpu().numpy()
        check_tokens(got, want[at.numpy()], [info[i] for i in at.tolist()], f"{shape}, {form}, from {lo}")


@pytest.mark.parametrize("rows,V,mean", [(150, 16_000, 16.0), (300, 16_000, -16.0), (60, 98_305, -3.0), (150, 16_000, 10.0), (300, 30_000, 5.0)])
def test_the_estimated_band_of_coarse_rows_holds_the_pivot(rows, V, mean):
    """Rows short enough for the lists to hold the few values of a band: it takes no exact select where the band holds the pivot.  (With
    edges at a rank's place in its bucket, where a single value lies anywhere, a third of such rows took one.)"""
    m = mods()
    g = torch.Generator().manual_seed(rows + V)
    n = torch.arange(rows)
    x = (torch.randn(rows, 1, V, generator=g) + mean).bfloat16()
    params = wl._params(rows, V, 0.5 + 0.7 * torch.rand(rows, generator=g), torch.full((rows,), V), 0.8 + 0.19 * torch.rand(rows, generator=g), torch.zeros(rows))
    u = wl.open_unit(g, rows, 1)
    got, st = m["draw"](x.cuda(), wl.sampler_params(params, V, "cuda"), None, u=u.cuda(), status=True, flags=_lib.KERNEL_AUTO)
    few = n[:: rows // 12].tolist()
    want, info = oracle_draw_rows(x[few].float().numpy(), {k: v[few] for k, v in np_params(params).items()}, None, u=u[few].numpy(), workers=1)
    check_tokens(got.cpu().numpy()[few], want, info, f"{rows} x {V} around {mean}")
    slow = int((st & _lib.ROW_SELECT_SLOW).ne(0).sum())
    print(f"{slow} of {rows} rows slow")
    assert slow <= rows // 30


@pytest.mark.parametrize("rows,V", [(300, 262_144), (300, 216_064)])
def test_bands_of_long_coarse_rows_fit_the_lists(rows, V):
    """A few values to a bucket of the histogram, 300 logits to a value: what the edges of a band move out by to end between values has
    to be made up for, or the lists of its warps overflow (5 of 160 rows of 262,144 did)."""
    m = mods()
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (torch.randn(rows, 1, V, generator=g, device="cuda") * 2).bfloat16()
    params = wl._params(rows, V, 0.8, V, 0.95, 0.0)
    u = wl.open_unit(torch.Generator().manual_seed(1), rows, 1)
    got, st = m["draw"](x, wl.sampler_params(params, V, "cuda"), None, u=u.cuda(), status=True, flags=_lib.KERNEL_AUTO)
    few = torch.arange(0, rows, rows // 8).tolist()
    want, info = oracle_draw_rows(x[few].float().cpu().numpy(), {k: v[few] for k, v in np_params(params).items()}, None, u=u[few].numpy(), workers=1)
    check_tokens(got.cpu().numpy()[few], want, info, f"{rows} x {V}")
    assert int((st & _lib.ROW_SELECT_SLOW).ne(0).sum()) <= 1

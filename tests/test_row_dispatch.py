"""The sampler's choice of a kernel by row count, vocabulary and type, at the edges of that choice and of the kernels' chunks, and
the small kernels that share a row among the CTAs of a cluster: against the CPU oracle."""
import numpy as np
import pytest
import torch

from colinfer_b200 import workloads as wl
from oracle import oracle as O

from test_gpu_parity import _check_logprobs, check_tokens, mods, np_params, verify_case

pytestmark = pytest.mark.gpu


def _case(rows, V, dtype, seed, levels=0, head=0):
    g = torch.Generator().manual_seed(seed)
    logits = (torch.randn(rows, 1, V, generator=g) * 2).to(dtype)
    if head:
        at = torch.randint(0, V, (rows, 1, head), generator=g)
        logits.scatter_(2, at, (logits.float().gather(2, at) + 8).to(dtype))
    if levels:                                                       # few distinct values: thousands of equal logits in a band
        logits = (torch.round(logits.float() * levels) / levels).to(dtype)
    T = torch.where(torch.arange(rows) % 7 == 6, 0.0, 0.4 + 0.8 * torch.rand(rows, generator=g))
    k = torch.tensor([V, 20, 100, 300, V])[torch.arange(rows) % 5].clamp_max(V)
    p = torch.where(torch.arange(rows) % 4 == 3, torch.tensor(1.0), 0.8 + 0.1999 * torch.rand(rows, generator=g))
    params = wl._params(rows, V, T, k, p, torch.where(torch.arange(rows) % 6 == 5, 0.02, 0.0))
    return g, logits, params, wl.open_unit(g, rows, 1)


# a cluster per row in few rows, one or two CTAs' worth of a row, more rows than SMs (148) and than they hold CTAs (296)
@pytest.mark.parametrize("rows,V,dtype,mask,hist,levels,head", [
    (1, 8191, "float32", True, 40, 0, 0), (17, 16385, "float32", False, 0, 0, 20), (36, 16384, "bfloat16", True, 0, 0, 0),
    (40, 65537, "float32", False, 64, 0, 0), (148, 512, "float32", False, 0, 0, 0), (149, 513, "float32", True, 0, 0, 0),
    (150, 511, "bfloat16", False, 300, 0, 0), (201, 8193, "float32", False, 700, 0, 20), (296, 1024, "bfloat16", True, 0, 0, 0),
    (298, 4099, "float32", True, 48, 0, 0), (151, 65536, "bfloat16", False, 0, 4, 0), (150, 65536, "bfloat16", False, 2500, 8, 0),
    (150, 65537, "float32", False, 0, 16, 0), (150, 229632, "bfloat16", False, 30, 0, 0), (150, 262144, "float32", False, 200, 0, 100),
    # long rows with histories: the last ones with an SM of their own, the first ones that share it
    (185, 216064, "float32", False, 200, 0, 0), (186, 216064, "float32", False, 200, 0, 0), (296, 216064, "bfloat16", False, 200, 0, 100),
    (297, 262144, "bfloat16", False, 200, 0, 0), (297, 280000, "bfloat16", False, 200, 0, 0),
])
def test_every_choice_of_kernel_draws_the_oracles_tokens(rows, V, dtype, mask, hist, levels, head):
    m = mods()
    g, logits, params, u = _case(rows, V, getattr(torch, dtype), rows * 7 + V, levels, head)
    sp = wl.sampler_params(params, V, "cuda")
    words = None
    if mask:
        allowed = torch.rand(rows, 1, V, generator=g) < 0.4
        allowed[..., V // 2] = True
        words = wl.pack_mask(allowed)
    history = None
    if hist:
        history = torch.randint(0, V, (rows, hist), generator=g, dtype=torch.int32)
        history[:, : hist // 4] = history[:, hist // 4: 2 * (hist // 4)]
        sp.set_history(history.cuda(), torch.full((rows,), hist, dtype=torch.int32, device="cuda"))
        sp._ensure_penalties()
        sp.repetition_penalty.fill_(1.2), sp.presence_penalty.fill_(0.3), sp.frequency_penalty.fill_(0.1)
    out = m["draw"](logits.cuda(), sp, None, u=u.cuda(), mask=None if words is None else words.cuda()).cpu().numpy()
    few = np.unique(np.linspace(0, rows - 1, 24 if V < 20000 else 8).astype(int))   # the oracle takes its time on long rows
    pr = {n: v[few] for n, v in np_params(params).items()}
    if hist:
        one = np.ones(len(few), np.float32)
        pr.update(repetition_penalty=np.float32(1.2) * one, presence_penalty=np.float32(0.3) * one, frequency_penalty=np.float32(0.1) * one)
    want, info = O.draw(logits[few].float().numpy(), pr, None, mask=None if words is None else words[few].numpy(),
                        history=None if history is None else history[few].numpy(),
                        hist_len=None if history is None else np.full(len(few), hist), u=u[few].numpy())
    check_tokens(out[few], want, info, f"{rows} x {V} {dtype}")


# one launch over target and draft rows: a cluster per row, more rows than SMs, and (100 rows) two launches
@pytest.mark.parametrize("B,k,V", [(2, 3, 8200), (20, 2, 700), (40, 2, 1027)])
def test_verify_over_both_sets_of_rows(B, k, V):
    g = torch.Generator().manual_seed(B + V)
    target = torch.randn(B, k + 1, V, generator=g) * 2
    draft = (target[:, :k] + torch.randn(B, k, V, generator=g) * 0.7).contiguous()
    params = wl._params(B, V, torch.where(torch.arange(B) % 5 == 0, 0.0, 0.9), torch.tensor([V, 40])[torch.arange(B) % 2], 0.95, 0.0)
    verify_case(target, draft, wl.open_unit(g, B, k), wl.open_unit(g, B, k), wl.open_unit(g, B, k + 1), params, V, k)


@pytest.mark.parametrize("rows,V,n_top", [(1, 32768, 20), (1, 33001, 32), (28, 32769, 5), (50, 16384, 20), (100, 8193, 1), (112, 8192, 0)])
def test_logprobs_of_rows_shared_by_a_cluster(rows, V, n_top):
    g = torch.Generator().manual_seed(rows + V)
    x = torch.randn(rows, V, generator=g) * 2
    x[0, 100:] = torch.round(x[0, 100:])                             # long runs of equal logits
    _check_logprobs(x, torch.randint(0, V, (rows,), generator=g).tolist(), n_top)


@pytest.mark.parametrize("V", [1, 127, 129, 16384, 16387, 50001])
def test_inverse_cdf_at_the_edges_of_the_warps_regions(V):
    m = mods()
    g = torch.Generator().manual_seed(V)
    P = torch.rand(9, V, generator=g) * (torch.rand(9, V, generator=g) < 0.3)
    P[:, V // 2] += 0.1
    P = P / P.sum(-1, keepdim=True)
    u = torch.rand(9, generator=g).clamp(1e-6, 1.0)
    got = m["inverse_cdf"](P.cuda(), u.cuda()).cpu().numpy()
    c = np.cumsum(P.numpy().astype(np.float64), -1)
    want = np.array([np.searchsorted(c[r], float(u[r]) * c[r, -1]) for r in range(9)])
    assert (got == want).all() and (P.numpy()[np.arange(9), got] > 0).all()


@pytest.mark.parametrize("k", [1, 31, 32, 33, 70])
def test_accept_of_long_drafts(k):
    m = mods()
    g = torch.Generator().manual_seed(k)
    B = 12
    tok = torch.randint(0, 50, (B, k + 1), generator=g)
    pred = torch.cat([tok[:, 1:], torch.randint(0, 50, (B, 1), generator=g)], 1)
    for b in range(1, B):
        pred[b, min(k, (b * 7) % (k + 2))] += 1
    stop = torch.full((B, 2), -1, dtype=torch.int64)
    stop[::3, 1] = tok[::3, (k + 1) // 2]
    active = (torch.arange(B) % 5 != 4).int()
    out, n = m["spec_accept"](pred.cuda(), tok.cuda(), stop.cuda(), active.cuda())
    want, wn = O.spec_accept(pred.numpy(), tok.numpy(), stop.numpy(), active.numpy())
    assert (out.cpu().numpy() == want).all() and (n.cpu().numpy() == wn).all()

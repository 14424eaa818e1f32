"""Timed cases of the logits -> token path: what an engine asks of this package at every decoding step, through the
package's public entry points, from one slot to a thousand.

listed() names the cases, draw() gives further ones of the same ranges, prepare() makes a case's inputs on the GPU from
a seed, run() is one pass, work() what a pass cannot do without, tolerance() how far another correct implementation of
the same precision may be off.

Kinds of a case:
  sample    draw() / sample(): one token per slot (rows = 1), or `rows` positions of a slot at once
  cycle     an exact-match speculative cycle: draw() over the k + 1 verified rows, spec_accept(), spec_advance()
  verify    spec_verify(): rejection verify of k drafts per slot against target and draft rows
  logprobs  logprobs_tensors(): log-probability of the emitted token and of the n_top most likely ones
  draft     lowrank_draft(): the greedy draft of a low-rank head (BF16 or NVFP4 lm_head)
  probs     processed_probs() of one slot's rows and inverse_cdf() on them

Options: dtype of the logits; mask = share of tokens a grammar allows (0: no mask); hist = length of the histories the
penalties count in (0: no penalties); head = tokens per row raised far above the rest (0: a flat row); filters = the
slots' sampling parameters ("mix": a third of the slots each with top_k 0, 20, 100, all with a top_p in [0.8, 1];
"single": temperature 0.7, top_k 50, top_p 0.9, min_p 0.05; "wide": temperature 1, top_k 1000, top_p 0.98, min_p 0.01;
"top_p": temperature 0.8, top_p 0.95; "plain": every other slot greedy, the rest temperature 1 without a filter).
"""
import math

import torch

from colinfer_b200.runtime.logprobs import logprobs_tensors
from colinfer_b200.runtime.sampler import SamplerParams, sample
from colinfer_b200.spec.accept import draw as draw_rows
from colinfer_b200.spec.accept import inverse_cdf, processed_probs
from colinfer_b200.spec.draft import lowrank_draft
from colinfer_b200.spec.verify import spec_accept, spec_advance, spec_verify

V_SMALL, V_MID, V_LARGE = 32_000, 151_936, 262_144     # vocabularies: the smallest in use, the usual one, the largest
MAX_LOGITS_BYTES = 1024 * V_MID * 4                     # the largest listed case: 1,024 fp32 rows
DRAFT_VOCAB, HIDDEN, CANDIDATES = 69_632, 2_560, 256    # the low-rank draft head


def _sample(slots, vocab, rows=1, dtype="float32", mask=0.0, hist=0, head=0, filters="mix"):
    return dict(kind="sample", slots=slots, rows=rows, vocab=vocab, dtype=dtype, mask=mask, hist=hist, head=head, filters=filters)


def _cycle(slots, k, vocab, dtype="float32"):
    return dict(kind="cycle", slots=slots, k=k, vocab=vocab, dtype=dtype)


def _verify(slots, k, vocab, dtype="float32"):
    return dict(kind="verify", slots=slots, k=k, vocab=vocab, dtype=dtype)


def _logprobs(rows, vocab, n_top, dtype="float32"):
    return dict(kind="logprobs", slots=rows, vocab=vocab, n_top=n_top, dtype=dtype)


def _draft(slots, fmt="bf16"):
    return dict(kind="draft", slots=slots, fmt=fmt)


def _probs(rows, vocab, filters):
    return dict(kind="probs", rows=rows, vocab=vocab, filters=filters)


def listed():
    return [
        # a single user's decoding step: one slot with every filter and penalties; all latency
        dict(_sample(1, V_MID, hist=512, filters="single"), name="sample_1"),
        # a few constrained slots (JSON output): a grammar that allows 2 % of the tokens, greedy or plain draws
        dict(_sample(4, V_MID, mask=0.02, filters="plain"), name="grammar_4"),
        # a busy engine's step: mixed requests with penalties over long histories
        dict(_sample(64, V_MID, hist=2048), name="sample_64"),
        # the benchmark's batch: the largest step
        dict(_sample(1024, V_MID, hist=2048), name="sample_1024"),
        # bf16 logits of the largest vocabulary under a grammar mask, peaked rows, a large top_k
        dict(_sample(512, V_LARGE, dtype="bfloat16", mask=0.3, head=100, filters="wide"), name="bf16_512"),
        # a vocabulary that is not padded: rows start at every alignment
        dict(_sample(201, 100_003), name="ragged_201"),
        # exact-match speculative decoding: 16 slots verify 7 drafts each, the accept and the bookkeeping behind it
        dict(_cycle(16, 7, V_MID), name="cycle_16x8"),
        # rejection verify for one user, and for a batch
        dict(_verify(1, 8, V_MID), name="verify_1x8"),
        dict(_verify(48, 4, V_MID), name="verify_48x4"),
        # requests that ask for logprobs with 20 alternatives
        dict(_logprobs(256, V_MID, 20), name="logprobs_256"),
        # what one speculative cycle drafts
        dict(_draft(16), name="draft_16"),
        # a host that wants the distribution itself: the rows of one verified slot, and its own draw on them
        dict(_probs(9, V_MID, "single"), name="probs_9"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _vocab(rng):
    v = _log_int(rng, V_SMALL, V_LARGE)
    return v if rng.random() < 0.3 else (v + 63) // 64 * 64             # most engines pad the lm_head, some do not


def draw(rng):
    kind = rng.choices(["sample", "cycle", "verify", "logprobs", "draft", "probs"], [10, 2, 3, 2, 2, 1])[0]
    V = _vocab(rng)
    dtype = "float32" if rng.random() < 0.7 else "bfloat16"
    most = MAX_LOGITS_BYTES // (V * (4 if dtype == "float32" else 2))     # rows
    if kind == "sample":
        slots = _log_int(rng, 1, min(1024, most))
        mask = rng.choice([0.0, 0.0, 0.02, 0.3, 0.95])
        hist = rng.choice([0, 1]) * _log_int(rng, 32, 2048)
        head = rng.choice([0, 0, 20, 100])
        return _sample(slots, V, dtype=dtype, mask=mask, hist=hist, head=head,
                       filters=rng.choice(["mix", "mix", "single", "wide", "top_p", "plain"]))
    if kind == "cycle":
        k = rng.randint(1, 15)
        return _cycle(_log_int(rng, 1, max(1, min(64, most // (k + 1)))), k, V, dtype)
    if kind == "verify":
        k = rng.randint(1, 8)
        return _verify(_log_int(rng, 1, max(1, min(128, most // (2 * k + 1)))), k, V, dtype)
    if kind == "logprobs":
        return _logprobs(_log_int(rng, 1, min(1024, most)), V, rng.choice([0, 1, 5, 20]), dtype)
    if kind == "draft":
        return _draft(_log_int(rng, 1, 256), rng.choice(["bf16", "nvfp4"]))
    return _probs(_log_int(rng, 1, 64), V, rng.choice(["single", "wide", "top_p"]))


# ------------------------------------------------------------------------------------------------ inputs
def _unit(g, *shape):
    """Uniforms in (0, 1], as the engine's Philox gives."""
    return (1.0 - torch.rand(*shape, generator=g, device="cuda")).clamp_min(1e-7)


def _logits(g, slots, rows, vocab, dtype, head=0):
    """N(0, 2^2), with `head` tokens of every row raised by 8: flat rows are the hardest to cut, peaked ones the usual."""
    x = torch.randn(slots, rows, vocab, generator=g, device="cuda").mul_(2.0)
    if head:
        at = torch.randint(0, vocab, (slots, rows, head), generator=g, device="cuda")
        x.scatter_(2, at, x.gather(2, at) + 8.0)
    return x if dtype == "float32" else x.to(torch.bfloat16)


def _mask(g, slots, rows, vocab, share):
    """int32 [slots, rows, ceil(vocab / 32)]: token t is bit t % 32 of word t // 32."""
    W = (vocab + 31) // 32
    bits = 1 << torch.arange(32, device="cuda")
    out = torch.empty(slots, rows, W, dtype=torch.int32, device="cuda")
    step = max(1, (1 << 26) // (rows * W * 32))
    for b in range(0, slots, step):
        ok = torch.rand(min(step, slots - b), rows, W, 32, generator=g, device="cuda") < share
        word = (ok * bits).sum(-1)
        out[b:b + step] = torch.where(word >= 1 << 31, word - (1 << 32), word).int()
    return out


def _params(g, slots, vocab, filters, hist=0):
    p = SamplerParams(slots, vocab, "cuda")
    p.seed.copy_(torch.randint(0, 1 << 40, (slots,), generator=g, device="cuda"))
    if filters == "mix":
        p.temperature.copy_(0.5 + 0.7 * torch.rand(slots, generator=g, device="cuda"))
        k = torch.tensor([vocab, 20, 100], dtype=torch.int32, device="cuda")
        p.top_k.copy_(k[torch.randint(0, 3, (slots,), generator=g, device="cuda")])
        p.top_p.copy_(0.8 + 0.2 * torch.rand(slots, generator=g, device="cuda"))
    elif filters == "single":
        p.temperature.fill_(0.7), p.top_k.fill_(50), p.top_p.fill_(0.9), p.log_min_p.fill_(math.log(0.05))
    elif filters == "wide":
        p.temperature.fill_(1.0), p.top_k.fill_(1000), p.top_p.fill_(0.98), p.log_min_p.fill_(math.log(0.01))
    elif filters == "top_p":
        p.temperature.fill_(0.8), p.top_p.fill_(0.95)
    else:
        p.temperature[1::2] = 1.0
        if slots == 1:
            p.temperature.fill_(1.0)
    if hist:
        p.set_history(torch.randint(0, vocab, (slots, hist), generator=g, device="cuda", dtype=torch.int32),
                      torch.full((slots,), hist, dtype=torch.int32, device="cuda"))
        p._ensure_penalties()
        p.repetition_penalty.fill_(1.1), p.presence_penalty.fill_(0.5), p.frequency_penalty.fill_(0.2)
    return p


_E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0]


def _lm_head(g, fmt, vocab, vocab_ids):
    """(weights, scales, global scale) of an lm_head [vocab, HIDDEN], and its rows vocab_ids in bf16."""
    if fmt == "bf16":
        w = torch.randn(vocab, HIDDEN, generator=g, device="cuda", dtype=torch.bfloat16).mul_(0.02)
        return w, None, None, w[vocab_ids]
    w = torch.randint(0, 256, (vocab, HIDDEN // 2), generator=g, device="cuda", dtype=torch.uint8)
    sf = (0.5 + torch.rand(vocab, HIDDEN // 16, generator=g, device="cuda")).to(torch.float8_e4m3fn)
    gs = 0.008
    pair = w[vocab_ids].long()
    table = torch.tensor(_E2M1, device="cuda", dtype=torch.bfloat16)
    rows = torch.stack([table[pair & 15], table[pair >> 4]], -1).view(vocab_ids.numel(), HIDDEN // 16, 16)
    rows = rows * (sf.view(torch.float8_e4m3fn)[vocab_ids].to(torch.bfloat16) * gs)[..., None]
    return w, sf, gs, rows.view(vocab_ids.numel(), HIDDEN)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + 17)
    kind = case["kind"]
    if kind == "sample":
        B, R, V = case["slots"], case["rows"], case["vocab"]
        x = _logits(g, B, R, V, case["dtype"], case["head"])
        s = dict(logits=x if R > 1 else x[:, 0], p=_params(g, B, V, case["filters"], case["hist"]),
                 pos=torch.randint(0, 4096, (B,), generator=g, device="cuda", dtype=torch.int32), mask=None)
        if case["mask"]:
            s["mask"] = _mask(g, B, R, V, case["mask"])
    elif kind == "cycle":
        B, k, V = case["slots"], case["k"], case["vocab"]
        x = _logits(g, B, k + 1, V, case["dtype"], 20)
        tok = x.argmax(-1)                                               # drafts that are mostly the target's own choice
        tok = torch.where(torch.rand(B, k + 1, generator=g, device="cuda") < 0.8, tok,
                          torch.randint(0, V, (B, k + 1), generator=g, device="cuda"))
        tok = torch.roll(tok, 1, 1).contiguous()                         # row r is fed tok[:, r] and predicts tok[:, r + 1]
        p = _params(g, B, V, "mix")
        p.temperature[::2] = 0.0                                         # half of the requests are greedy
        s = dict(logits=x, p=p, tok=tok, stop=torch.randint(0, V, (B, 4), generator=g, device="cuda"),
                 active=torch.ones(B, dtype=torch.int32, device="cuda"), y=tok[:, 0].clone(),
                 history=torch.randint(0, V, (B, 2048), generator=g, device="cuda", dtype=torch.int32),
                 hist_len=torch.randint(16, 2048, (B,), generator=g, device="cuda", dtype=torch.int32),
                 pos=torch.randint(0, 4096, (B,), generator=g, device="cuda"))
    elif kind == "verify":
        B, k, V = case["slots"], case["k"], case["vocab"]
        target = _logits(g, B, k + 1, V, "float32")
        draft = target[:, :k] + torch.randn(B, k, V, generator=g, device="cuda") * 0.5
        ids = (draft / 0.8 - (-_unit(g, B, k, V).log()).clamp_min(1e-30).log()).argmax(-1)   # drawn from the draft model
        dt = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
        s = dict(target=target.to(dt), draft=draft.to(dt), ids=ids, p=_params(g, B, V, "top_p"), ua=_unit(g, B, k), us=_unit(g, B, k + 1))
    elif kind == "logprobs":
        x = _logits(g, case["slots"], 1, case["vocab"], case["dtype"], 20)[:, 0]
        s = dict(rows=x, toks=torch.randint(0, case["vocab"], (case["slots"],), generator=g, device="cuda"), n_top=case["n_top"])
    elif kind == "draft":
        N = case["slots"]
        ids = torch.randperm(V_MID, generator=g, device="cuda")[:DRAFT_VOCAB]
        w, sf, gs, rows = _lm_head(g, case["fmt"], V_MID, ids)
        x = torch.randn(N, HIDDEN, generator=g, device="cuda", dtype=torch.bfloat16)
        ap = (x @ rows.T).float() + 0.3 * torch.randn(N, DRAFT_VOCAB, generator=g, device="cuda")
        s = dict(ap=ap.contiguous(), x=x, w=w, sf=sf, gs=gs, ids=ids)
    else:
        R, V = case["rows"], case["vocab"]
        s = dict(logits=_logits(g, 1, R, V, "float32")[0], p=_params(g, 1, V, case["filters"]), u=_unit(g, R))
    s["kind"] = kind
    return s


def run(state):
    s, kind = state, state["kind"]
    if kind == "sample":
        if s["logits"].dim() == 2:
            return sample(s["logits"], s["p"], s["pos"], mask=s["mask"])
        return draw_rows(s["logits"], s["p"], s["pos"], mask=s["mask"])
    if kind == "cycle":
        pred = draw_rows(s["logits"], s["p"], s["pos"])
        out_tok, n = spec_accept(pred, s["tok"], s["stop"], s["active"])
        spec_advance(out_tok, n, s["y"], s["history"], s["hist_len"], s["pos"])
        return dict(pred=pred, out_tok=out_tok, n=n, y=s["y"], history=s["history"], hist_len=s["hist_len"], pos=s["pos"])
    if kind == "verify":
        return spec_verify(s["target"], s["draft"], s["ids"], s["p"], s["ua"], s["us"])
    if kind == "logprobs":
        return logprobs_tensors(s["rows"], s["toks"], s["n_top"])
    if kind == "draft":
        return lowrank_draft(s["ap"], s["x"], s["w"], s["ids"], s["sf"], s["gs"], n_cands=CANDIDATES)
    p = s["p"]
    P = processed_probs(s["logits"], p.temperature, p.top_k, p.top_p, p.log_min_p)
    return P, inverse_cdf(P, s["u"])


def work(case):
    """Each input read once, each output written once; a multiply-add per element of a dot product.  (The selection
    itself is comparisons, an exponential per logit at most.)"""
    kind = case["kind"]
    elt = 2 if case.get("dtype") == "bfloat16" else 4
    if kind == "sample":
        n, V = case["slots"] * case["rows"], case["vocab"]
        row = V * elt + (4 * ((V + 31) // 32) if case["mask"] else 0) + 8
        return {"bytes": n * row + case["slots"] * (4 * case["hist"] + 32), "flops": 0}
    if kind == "cycle":
        B, k1, V = case["slots"], case["k"] + 1, case["vocab"]
        return {"bytes": B * (k1 * (V * elt + 8 * 3) + 8 * k1 + 100), "flops": 0}
    if kind == "verify":
        B, k, V = case["slots"], case["k"], case["vocab"]
        return {"bytes": B * ((2 * k + 1) * V * elt + 8 * (3 * k + 2) + 36), "flops": 0}
    if kind == "logprobs":
        return {"bytes": case["slots"] * (case["vocab"] * elt + 12 + 12 * case["n_top"]), "flops": 0}
    if kind == "draft":
        row = HIDDEN * 2 if case["fmt"] == "bf16" else HIDDEN // 2 + HIDDEN // 16
        return {"bytes": case["slots"] * (DRAFT_VOCAB * 4 + CANDIDATES * (row + 8) + HIDDEN * 2 + 12),
                "flops": 2.0 * case["slots"] * CANDIDATES * HIDDEN}
    return {"bytes": case["rows"] * (case["vocab"] * 8 + 12), "flops": 0}


def tolerance(case):
    """Tokens are whole numbers: they differ only where a row's uniform (or top-p target) lies within the rounding of the
    fp32 exponentials of a step of its distribution.  Probabilities and logprobs: fp32 exponentials and sums."""
    if case["kind"] == "logprobs":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.001}
    if case["kind"] == "draft":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] == "probs":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.002}
    return {"differ": 0.002}

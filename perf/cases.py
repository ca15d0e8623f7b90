"""Performance cases of the chunked delta-rule layer: the calls that training and serving programs make, from one token per
sequence to 64k packed tokens, with the option sets of the benchmark configurations and of the tests.

A case is a dict of plain values:

  op        "kda": ``chunk_kda`` (one decay per token, v-head and key channel), "gdr": ``chunk_gated_delta_rule`` (one per
            token and v-head)
  train     forward and backward with dense upstream gradients, else forward only under ``no_grad``
  rows, tokens, docs, doc_seed
            ``rows`` x ``tokens`` with docs = 0; docs > 0: one row of ``tokens`` packed documents with lognormal lengths (median
            ``docs``, sigma 1), cut at multiples of ``row_len`` and addressed by ``cu_seqlens``
  HK, HV    q/k heads and v-heads; dtype of q, k, v and of the norm's gate; gate_dtype of the raw gate
  gate, beta, beta_scale, l2, norm, state_in, state_out, v_first
            the options of the call (norm = activation of the gated RMSNorm epilogue or "")
"""
import math

import numpy as np
import torch

from mogankda_b200 import chunk_gated_delta_rule, chunk_kda

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
#: the largest listed case: 65 536 tokens x 32 v-heads
MOST_TOKEN_HEADS = 65536 * 32


def _case(**kw):
    c = dict(op="kda", train=True, rows=1, tokens=0, docs=0, doc_seed=0, row_len=0, HK=16, HV=32, dtype="bf16", gate_dtype="fp32",
             gate="eda", beta="sigmoid", beta_scale=1.0, l2=True, norm="", state_in=False, state_out=False, v_first=False)
    c.update(kw)
    return c


def listed():
    return [
        # one more token for each of eight running sequences: state in, state out (the smallest call: latency and launches)
        _case(name="step_b8_t1", train=False, rows=8, tokens=1, gate="kimi", norm="silu", state_in=True, state_out=True),
        # a short prompt of one user, not a multiple of the chunk
        _case(name="prompt_t77", train=False, tokens=77, HK=8, HV=16, beta_scale=2.0, norm="silu", state_out=True),
        # a serving batch: ragged prompts packed together, each continuing from a state of its own
        _case(name="prefill_packed_6k", train=False, tokens=6001, docs=200, doc_seed=3, beta_scale=2.0, norm="silu",
              state_in=True, state_out=True, v_first=True),
        # one long prompt of odd length
        _case(name="prefill_long_32k", train=False, tokens=32749, gate="kimi", norm="sigmoid", state_out=True),
        # scalar-gate prompts of a serving batch, equal lengths
        _case(name="gdr_prefill_4x2k", op="gdr", train=False, rows=4, tokens=2000, HK=16, HV=16, gate="precomputed",
              beta="precomputed", l2=True, state_in=True, state_out=True, v_first=True),
        # the small fp32 configuration that is also run on the CPU: T=256, HK2/HV4, precomputed gate
        _case(name="train_fp32_t256", tokens=256, HK=2, HV=4, dtype="fp32", gate="precomputed", beta="precomputed", l2=False,
              state_out=True),
        # fp16 fine-tuning batch with a 16-bit raw gate and rows of 1000 tokens
        _case(name="train_fp16_4x1000", rows=4, tokens=1000, HK=4, HV=8, dtype="fp16", gate_dtype="fp16", gate="gdn", norm="sigmoid",
              state_in=True),
        # the 1B-shape layer, 8192 tokens in a few documents
        _case(name="train_1b_8k", tokens=8192, docs=3000, doc_seed=21, HK=8, HV=16, beta_scale=2.0, norm="silu"),
        # very short documents (chat turns): most chunks are not full
        _case(name="train_short_docs_8k", tokens=8191, docs=60, doc_seed=5, HK=16, HV=16, gate="kimi", norm="silu"),
        # the headline configuration: packed short documents, 64k tokens
        _case(name="train_packed_64k", tokens=65536, docs=500, doc_seed=0, row_len=8192, beta_scale=2.0, norm="silu"),
        # one document of 64k tokens
        _case(name="train_long_64k", tokens=65536, gate="kimi"),
        # the scalar-gate configuration with initial and final states in [V, K] layout
        _case(name="gdr_train_4x16k", op="gdr", rows=4, tokens=16384, HK=16, HV=16, gate="precomputed", beta="precomputed", l2=False,
              state_in=True, state_out=True, v_first=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: an entry point, a direction and a size over the whole range, the options drawn independently."""
    op = rng.choice(("kda", "kda", "gdr"))
    train = rng.random() < 0.6
    HK = rng.choice((1, 2, 4, 8, 16, 16))
    HV = HK * rng.choice((1, 2, 2, 4)) if HK <= 8 else HK * rng.choice((1, 2))
    most = min(65536, MOST_TOKEN_HEADS // HV)
    shape = rng.choice(("one", "rows", "packed", "packed") if train else ("one", "rows", "packed", "step"))
    kw = dict(op=op, train=train, HK=HK, HV=HV, doc_seed=rng.randrange(1 << 20))
    if shape == "step":
        kw.update(rows=_log_int(rng, 1, 64), tokens=rng.choice((1, 1, 2, 4)))
    elif shape == "rows":
        kw["rows"] = rng.choice((2, 3, 4, 8))
        kw["tokens"] = _log_int(rng, 16, most // kw["rows"])
    elif shape == "one":
        kw["tokens"] = _log_int(rng, 16, most)
    else:
        kw["tokens"] = _log_int(rng, 256, most)
        # many very short documents in the largest batches would cost more than the largest listed case
        kw["docs"] = _log_int(rng, 60 if kw["tokens"] * HV <= MOST_TOKEN_HEADS // 4 else 400, 4000)
    kw["dtype"] = rng.choice(("bf16", "bf16", "bf16", "fp16", "fp32"))
    if kw["dtype"] == "fp32" and kw["tokens"] * kw.get("rows", 1) * HV > MOST_TOKEN_HEADS // 4:
        kw["dtype"] = "bf16"
    if op == "gdr":
        kw.update(gate="precomputed", beta="precomputed", l2=rng.random() < 0.5)
    else:
        kw.update(gate=rng.choice(("eda", "eda", "kimi", "kimi", "gdn", "precomputed")), beta=rng.choice(("sigmoid", "sigmoid", "precomputed")),
                  beta_scale=rng.choice((1.0, 2.0)), l2=rng.random() < 0.8, norm=rng.choice(("silu", "silu", "sigmoid", "")))
        if kw["gate"] != "precomputed" and rng.random() < 0.25:
            kw["gate_dtype"] = "bf16"
    if kw["beta"] == "precomputed":
        kw["beta_scale"] = 1.0
    few = kw.get("docs", 0) == 0 or kw["tokens"] // kw["docs"] <= 64
    kw["state_in"] = few and (shape == "step" or rng.random() < 0.4)
    kw["state_out"] = few and (shape == "step" or not train or rng.random() < 0.3)
    kw["v_first"] = (kw["state_in"] or kw["state_out"]) and rng.random() < 0.5
    return _case(**kw)


def _bounds(c):
    """Boundaries of the packed documents, None without packing."""
    if not c["docs"]:
        return None
    g, cu = np.random.RandomState(c["doc_seed"]), [0]
    row = c["row_len"] or c["tokens"]
    while cu[-1] < c["tokens"]:
        end = min((cu[-1] // row + 1) * row, c["tokens"])
        cu.append(min(cu[-1] + max(int(g.lognormal(math.log(c["docs"]), 1.0)), 1), end))
    return cu


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, T, HK, HV = c["rows"], c["tokens"], c["HK"], c["HV"]
    dt, per_channel = DTYPES[c["dtype"]], c["op"] == "kda"
    cu = _bounds(c)
    N = B if cu is None else len(cu) - 1

    def r(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    q, k = r(B, T, HK, 128), r(B, T, HK, 128)
    if not c["l2"]:          # the layer normalises q and k itself before the call
        q, k = torch.nn.functional.normalize(q, dim=-1), torch.nn.functional.normalize(k, dim=-1)
    x = r(B, T, HV, 128) if per_channel else r(B, T, HV)
    t = dict(q=q.to(dt), k=k.to(dt), v=r(B, T, HV, 128).to(dt))
    del q, k
    if c["gate"] == "precomputed":          # natural-log decay per token, in [-5, 0]
        t["g"] = -0.5 * torch.sigmoid(x) if per_channel else torch.clamp(-torch.exp(0.1 * r(HV)) * torch.nn.functional.softplus(x), min=-5.0)
    else:
        t["g"] = x.to(DTYPES[c["gate_dtype"]])
        t["A_log"], t["dt_bias"] = 0.1 * r(HV), 0.1 * r(HV, 128)
    del x
    t["beta"] = r(B, T, HV) if c["beta"] == "sigmoid" else torch.sigmoid(r(B, T, HV))
    if c["state_in"]:
        t["h0"] = 0.02 * r(N, HV, 128, 128)
    if c["norm"]:
        t["norm_w"], t["norm_gate"] = 1.0 + 0.1 * r(128), r(B, T, HV, 128).to(dt)
    s = dict(case=c, leaves=t, cu=None if cu is None else torch.tensor(cu, dtype=torch.int32, device="cuda"))
    if c["train"]:
        for x in t.values():
            x.requires_grad_(True)
        s["do"] = r(B, T, HV, 128).to(torch.float32 if c["norm"] else dt)
        s["dht"] = 0.1 * r(N, HV, 128, 128) if c["state_out"] else None
    return s


def _forward(s):
    c, t = s["case"], s["leaves"]
    if c["op"] == "gdr":
        return chunk_gated_delta_rule(t["q"], t["k"], t["v"], t["g"], t["beta"], initial_state=t.get("h0"), output_final_state=c["state_out"],
                                      use_qk_l2norm_in_kernel=c["l2"], cu_seqlens=s["cu"], state_v_first=c["v_first"])
    norm = dict(weight=t["norm_w"], gate=t["norm_gate"], act=c["norm"], eps=1e-6) if c["norm"] else None
    return chunk_kda(t["q"], t["k"], t["v"], t["g"], t["beta"], initial_state=t.get("h0"), output_final_state=c["state_out"],
                     cu_seqlens=s["cu"], state_v_first=c["v_first"], gate_mode=c["gate"], A_log=t.get("A_log"), dt_bias=t.get("dt_bias"),
                     lower_bound=-5.0, beta_mode=c["beta"], beta_scale=c["beta_scale"], use_qk_l2norm_in_kernel=c["l2"], output_norm=norm)


def run(state):
    if not state["case"]["train"]:
        with torch.no_grad():
            o, ht = _forward(state)
        return dict(o=o, ht=ht)
    o, ht = _forward(state)
    outs, ups = ((o, ht), (state["do"], state["dht"])) if ht is not None else ((o,), (state["do"],))
    grads = torch.autograd.grad(outs, list(state["leaves"].values()), ups)
    res = {"d" + n: d for n, d in zip(state["leaves"], grads)}
    res.update(o=o.detach(), ht=None if ht is None else ht.detach())
    return res


def work(case):
    """Each input read once, each output written once (a backward pass: upstream gradients in, one gradient per input out), and the
    chunk-algebra products at 64 tokens per chunk, counted once (no precision split, no recomputation)."""
    c = case
    n, HK, HV = c["rows"] * c["tokens"], c["HK"], c["HV"]
    cu = _bounds(c)
    N = c["rows"] if cu is None else len(cu) - 1
    e, eg = DTYPES[c["dtype"]].itemsize, DTYPES[c["gate_dtype"]].itemsize
    eo = 4 if c["norm"] else e
    gate = n * HV * (128 if c["op"] == "kda" else 1) * (4 if c["gate"] == "precomputed" else eg)
    inputs = n * (2 * HK + HV) * 128 * e + gate + n * HV * 4
    inputs += n * HV * 128 * e if c["norm"] else 0
    inputs += N * HV * 65536 if c["state_in"] else 0
    outputs = n * HV * 128 * eo + (N * HV * 65536 if c["state_out"] else 0)
    if c["train"]:
        return {"bytes": 2 * (inputs + outputs), "flops": 573440 * n * HV}
    return {"bytes": inputs + outputs, "flops": 163840 * n * HV}


def tolerance(case):
    """16-bit inputs: about two roundings of a 16-bit store (2^-9 rms each) in the results that are stored that way; the 32-bit results
    of the same call are sums of products with 16 mantissa bits per operand (bf16 high and low halves), the parameter gradients sums over
    all tokens with heavy cancellation.  fp32 inputs: those products, about 2e-5 each, through the chain of products of a chunk and of
    the backward pass."""
    return {"rel": 5e-3} if case["dtype"] != "fp32" else {"rel": 5e-4}

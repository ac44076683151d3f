"""Workloads of the stick-breaking attention operators, from single short prompts to long-context training steps.

Every case is one call of a public operator (``sb_attn_varlen``, ``sb_attn`` or their ``_fused`` forms), forward only
or forward and backward.  Sizes are those of the package's benchmark configurations, its length sweep and its tests.

The score distribution decides how far back a query looks, so it is part of a case (``data``):

* ``normal``     q, k ~ N(0, std^2): the benchmark configurations.  About one bit of stick is broken off per key, so the
                 stick is used up (the remainder is below the smallest fp32 number) some 110 to 130 keys before the query.
* ``reference``  the shifted 0.25 recipe of the reference operator's tests: negative scores, several hundred keys.
* ``spread``     a trained head that spreads its stick over the whole context: scores around -log(longest sequence), so
                 no key's weight vanishes.
"""
import math

import numpy as np
import torch

import stickbreaking_attention_b200 as sb

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}

# form: "packed" (heads, tokens, d) with cumulative sequence ends, or "fixed" (batch, heads, tokens, d)
# shape: packed: `seqs` sequences with lengths from `low` to `high` (`spacing`: how they are drawn); fixed: `seqs` x `high`
DEFAULTS = {"form": "packed", "fused": False, "train": True, "dtype": "bf16", "heads": 16, "head_dim": 128, "seqs": 1,
            "low": 0, "high": 1, "spacing": "equal", "tokens": 0, "data": "spread", "std": 1.0, "attend_current": False,
            "zero_start": False, "token_major": False}


def _case(**kw):
    return {**DEFAULTS, **kw}


def listed():
    return [
        # scoring one short prompt: a single small forward call, where the call itself is most of the time
        _case(name="prompt_forward", form="fixed", train=False, dtype="fp16", heads=8, head_dim=64, high=200, data="normal"),
        # the fp32 configuration the operator is validated on: four ragged sequences, 960 tokens
        _case(name="packed_fp32_small", dtype="fp32", heads=4, head_dim=64, seqs=4, low=64, high=512, spacing="doubling",
              data="normal"),
        # a fine-tuning micro-batch of short texts, every token also attending to itself
        _case(name="finetune_small", heads=12, head_dim=64, seqs=8, low=16, high=256, spacing="uniform", attend_current=True,
              zero_start=True),
        # the odd sizes of the reference operator's test grid: 7 heads, 500 tokens, head size 50
        _case(name="odd_head_fixed", form="fixed", heads=7, head_dim=50, high=500, data="reference"),
        # an fp32 training step (debugging and numerics work)
        _case(name="fixed_fp32_train", form="fixed", dtype="fp32", heads=8, head_dim=64, seqs=2, high=1024),
        # the headline configuration: 16 heads, 8 sequences of 2048 tokens
        _case(name="headline_packed", seqs=8, high=2048, data="normal"),
        # the length sweep's first point: batch 4, 12 heads, activations kept token-major and passed as permuted views
        _case(name="sweep_fixed_4096", form="fixed", heads=12, seqs=4, high=4096, token_major=True),
        # head size 64 through the fused operator o + rem * v, token-major as well
        _case(name="fused_64", fused=True, dtype="fp16", head_dim=64, seqs=8, high=2048, token_major=True),
        # packed documents of lognormal length filling 65536 tokens
        _case(name="skewed_packed", heads=32, seqs=0, low=64, high=16384, spacing="lognormal", tokens=65536, zero_start=True),
        # prefill of many short requests at once, forward only (a quarter of the 4096-sequence configuration)
        _case(name="short_serving", train=False, heads=32, head_dim=64, seqs=1024, low=128, high=512, spacing="uniform",
              data="normal"),
        # prefill of one long prompt, forward only
        _case(name="prefill_16k", form="fixed", train=False, heads=32, high=16384),
        # one rank's share (2 of 16 heads) of the 131072-token training configuration
        _case(name="long_context", heads=2, high=131072, data="normal", std=0.5),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        form = rng.choice(["packed", "packed", "fixed"])
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
        head_dim = rng.choice([64, 128] if dtype == "fp32" else [64, 128, 128, 50, 72, 96])
        exact = dtype == "fp32" or head_dim % 8 != 0         # CUDA-core arithmetic: smaller sizes are what it is used for
        case = _case(form=form, fused=rng.random() < 0.2, train=rng.random() < 0.7, dtype=dtype, head_dim=head_dim,
                     heads=rng.choice([1, 2, 4, 7, 8, 12, 16, 32]), data=rng.choice(["normal", "spread", "spread", "reference"]),
                     attend_current=rng.random() < 0.2, token_major=rng.random() < 0.3)
        case["high"] = _log_uniform(rng, 40, 2048 if exact else 32768)
        tokens = max(case["high"], _log_uniform(rng, 100, 4096 if exact else 131072))
        if form == "fixed":
            case["seqs"] = max(1, tokens // case["high"])
        else:
            case["zero_start"] = rng.random() < 0.5
            case["spacing"] = rng.choice(["equal", "uniform", "lognormal"])
            case["low"] = max(1, case["high"] // rng.choice([2, 8, 32]))
            if case["spacing"] == "lognormal":
                case["tokens"], case["seqs"] = tokens, 0
            else:
                case["seqs"] = max(1, 2 * tokens // (case["high"] + case["low"]))
        dense = (7 if case["train"] else 2) * head_dim * case["heads"] * sum(n * n for n in lengths(case))
        if dense <= (8e9 if exact else 6e12):
            return case


def lengths(case):
    """The sequence lengths of a case (the same for every seed: a data loader's bucket)."""
    lo, hi, n = case["low"], case["high"], case["seqs"]
    if case["form"] == "fixed" or case["spacing"] == "equal":
        return [hi] * n
    if case["spacing"] == "doubling":
        return [hi // 4, hi // 2, lo, hi][:n]
    gen = np.random.default_rng(1)
    if case["spacing"] == "uniform":
        return [int(x) for x in gen.integers(lo, hi + 1, n)]
    out, left = [], case["tokens"]                            # lognormal, median 1024 (or the middle of the range), sigma 1
    median = min(1024.0, math.sqrt(lo * hi))
    while left > 0:
        x = int(np.clip(gen.lognormal(math.log(median), 1.0), lo, hi))
        out.append(min(x, left))
        left -= out[-1]
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, d, heads = DTYPES[case["dtype"]], case["head_dim"], case["heads"]
    lens = lengths(case)
    lead = (case["seqs"], case["high"]) if case["form"] == "fixed" else (sum(lens),)

    def tensor(shift=0.0, scale=1.0):
        # token-major activations (…, tokens, heads, d) are handed over as permuted views, as a projection leaves them
        shape = (*lead, heads, d) if case["token_major"] else (*lead[:-1], heads, lead[-1], d)
        x = torch.randn(shape, generator=gen, device="cuda", dtype=dtype).mul_(scale).add_(shift)
        return x.transpose(-2, -3) if case["token_major"] else x

    if case["data"] == "normal":
        q, k, v = (tensor(scale=case["std"]) for _ in range(3))
    elif case["data"] == "reference":
        q, k, v = tensor(0.25, 0.25), tensor(-0.25, 0.25), tensor(scale=0.25)
    else:
        # <q, k> / sqrt(d) ~ N(-shift^2 sqrt(d), 1 + 2 shift^2); the last term undoes the widening of the exponential's mean
        target = math.log(max(max(lens), 4)) + 0.5
        shift = math.sqrt(target / (math.sqrt(d) - 1))
        q, k, v = tensor(shift), tensor(-shift), tensor()
    state = {"case": case, "q": q, "k": k, "v": v}
    if case["form"] == "packed":
        ends = torch.tensor(lens, dtype=torch.int64).cumsum(0)
        if case["zero_start"]:
            ends = torch.cat((torch.zeros(1, dtype=torch.int64), ends))
        state["cu_seqlens"] = ends.to(torch.int32).cuda()
        state["max_seqlens"] = max(lens)
    if case["train"]:
        for name in ("q", "k", "v"):
            state[name].requires_grad_(True)
        state["do"] = tensor()
        if not case["fused"]:
            state["drem"] = torch.randn(q.shape[:-1], generator=gen, device="cuda", dtype=dtype)
    return state


def _forward(state):
    case, q, k, v = state["case"], state["q"], state["k"], state["v"]
    if case["form"] == "packed":
        op = sb.sb_attn_varlen_fused if case["fused"] else sb.sb_attn_varlen
        return op(q, k, v, state["cu_seqlens"], state["max_seqlens"], zero_start=case["zero_start"],
                  attend_current=case["attend_current"])
    op = sb.sb_attn_fused if case["fused"] else sb.sb_attn
    return op(q, k, v, attend_current=case["attend_current"])


def run(state):
    case = state["case"]
    if not case["train"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    outs, grads = (out, state["do"]) if case["fused"] else (out, (state["do"], state["drem"]))
    dq, dk, dv = torch.autograd.grad(outs, (state["q"], state["k"], state["v"]), grads)
    return {"out": out if case["fused"] else list(out), "dq": dq, "dk": dk, "dv": dv}


# bits of stick broken off per key, E[log2(1 + exp(z))], for the inputs whose stick does not last
def _reach(case):
    if case["data"] == "spread":
        return math.inf
    if case["data"] == "normal":
        mean, var = 0.0, case["std"] ** 4
    else:
        s = math.sqrt(case["head_dim"])
        mean, var = -0.0625 * s, 0.0625 ** 2 * 3
    z = np.linspace(-6, 6, 241)
    w = np.exp(-z * z / 2)
    bits = float((w * np.log2(1 + np.exp(mean + math.sqrt(var) * z))).sum() / w.sum())
    return 126.0 / bits


def work(case):
    """Bytes: inputs once, outputs once.  Operations: the forward's two products and the backward's five (scores again,
    dP, dQ, dK, dV) over the (query, key) pairs whose weight is not exactly zero in fp32."""
    lens = lengths(case)
    esize = 4 if case["dtype"] == "fp32" else 2
    tokens, heads, d = sum(lens), case["heads"], case["head_dim"]
    reach = _reach(case)
    pairs = sum(n * n / 2 if n <= reach else reach * reach / 2 + (n - reach) * reach for n in lens)
    row, rem = tokens * heads * d * esize, 0 if case["fused"] else tokens * heads * esize
    if not case["train"]:
        return {"bytes": 4 * row + rem, "flops": 4.0 * d * heads * pairs}
    return {"bytes": 8 * row + 2 * rem, "flops": 14.0 * d * heads * pairs}


def tolerance(case):
    # 16-bit tensors: the attention weights and the score gradients are rounded to the tensors' type before the second
    # products, and so are the results; fp32: sums of a few hundred to a few thousand fp32 terms
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 2e-5}[case["dtype"]]}

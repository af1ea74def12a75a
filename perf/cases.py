"""The attention work that a user of this package has it do, as cases that can be timed and compared.

Two families, both through the public entry points.  ``sdpa``: ScaledDotProductAttention on dense tensors, as a model
without a paged cache calls it.  ``paged``: one step of a continuous-batching loop through ``PagedAttentionOp`` - the
new tokens' K/V rows are stored into the block pool, then every new token attends over its sequence's cached context
(optionally with the operator's score output).  ``listed`` names twelve of them, ``draw`` gives others of the same
ranges.
"""
import math
import random

import torch

import openvino_contrib_b200 as b2a

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "u8": torch.uint8}
BLOCK = 16


def _sdpa(name, dtype, b, hq, hkv, sq, skv, d, causal, mask="none", layout="bhsd"):
    """mask: "none", "bool" or "add" (a [B, 1, 1, Skv] padding mask: every sequence of the batch has its own length).
    layout: "bhsd" dense tensors, "bshd" [B, S, H, D] storage viewed as [B, H, S, D] (what a projection layer
    writes), "cache" K and V are the first Skv rows of a longer preallocated cache."""
    c = dict(family="sdpa", dtype=dtype, b=b, hq=hq, hkv=hkv, sq=sq, skv=skv, d=d, causal=causal, mask=mask, layout=layout)
    return dict(c, name=name) if name else c


def _paged(name, dtype, kv, hq, hkv, decode, ctx_lo, ctx_hi, prefill=0, new_lo=0, new_hi=0, past_hi=0, capacity=0,
           lens_seed=1, scores=False):
    """`decode` sequences with one new token and contexts uniform in [ctx_lo, ctx_hi]; `prefill` sequences with
    uniform [new_lo, new_hi] new tokens behind a past of up to past_hi tokens (0: a fresh prompt).  The lengths follow
    from lens_seed alone.  capacity: the longest context the operator is built for.  D = 128, 16-token blocks."""
    c = dict(family="paged", dtype=dtype, kv=kv, hq=hq, hkv=hkv, decode=decode, ctx_lo=ctx_lo, ctx_hi=ctx_hi, prefill=prefill,
             new_lo=new_lo, new_hi=new_hi, past_hi=past_hi, capacity=capacity, lens_seed=lens_seed, scores=scores)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small float32 attention: the single operator of a functional test, where latency counts
        _sdpa("sdpa_f32_short", "f32", 1, 8, 8, 256, 256, 64, True),
        # a batch of padded sequences through an encoder block of head size 64, activations in [B, S, H, D]
        _sdpa("sdpa_encoder", "f16", 8, 16, 16, 512, 512, 64, False, "bool", "bshd"),
        # one prompt of odd length
        _sdpa("sdpa_prefill_odd", "f16", 1, 32, 8, 777, 777, 128, True, "none", "bshd"),
        # the benchmark's causal prefill of four 4096-token prompts
        _sdpa("sdpa_prefill", "bf16", 4, 32, 8, 4096, 4096, 128, True),
        # token generation of a stateful model: one query row over a dense cache, left-padded batch, odd length
        _sdpa("sdpa_cached_decode", "bf16", 8, 32, 8, 1, 3003, 128, False, "add", "cache"),
        # an interactive session or two: the smallest serving step, launch latency and host work
        _paged("paged_decode_few", "f16", "u8", 32, 8, 2, 300, 900, capacity=4096, lens_seed=5),
        # the benchmark's serving step: 64 sequences of uneven length
        _paged("paged_decode", "f16", "u8", 32, 8, 64, 512, 8192, capacity=8192, lens_seed=2),
        # the benchmark's long contexts, eight query heads per KV head
        _paged("paged_decode_long", "f16", "u8", 64, 8, 16, 32768, 32768, capacity=32768, lens_seed=3),
        # serving with an unquantised cache
        _paged("paged_decode_bf16_cache", "bf16", "bf16", 32, 8, 32, 256, 4096, capacity=4096, lens_seed=6),
        # chunked prefill: a few sequences continue their prompts behind what is cached already
        _paged("paged_prefill_chunks", "f16", "u8", 32, 8, 0, 0, 0, prefill=3, new_lo=400, new_hi=1100, past_hi=3000,
               capacity=4096, lens_seed=7),
        # the benchmark's mixed step: eight fresh 1024-token prompts beside 120 generating sequences
        _paged("paged_mixed", "bf16", "u8", 32, 8, 120, 256, 4096, prefill=8, new_lo=1024, new_hi=1024, capacity=4096,
               lens_seed=4),
        # generation with the score output that a cache-eviction policy accumulates
        _paged("paged_scores", "f16", "u8", 32, 8, 32, 512, 4096, capacity=4096, lens_seed=8, scores=True),
    ]


# the largest listed case in either unit: a drawn case stays below both
MAX_FLOPS, MAX_BYTES = 5.5e11, 1.12e9


def _log_int(rng, lo, hi):
    """Spread over the logarithm; half of them a multiple of nothing in particular."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if rng.random() < 0.5 else max(lo, n // 16 * 16)


def _draw_once(rng):
    kind = rng.choice(["f32", "encoder", "prefill", "prefill", "cached", "decode", "decode", "decode", "decode16",
                       "chunks", "mixed", "scores"])
    half = rng.choice(["f16", "bf16"])
    hq, hkv = rng.choice([(32, 8), (32, 8), (64, 8), (16, 4), (8, 8)])
    if kind == "f32":
        s, h = _log_int(rng, 32, 1024), rng.choice([4, 8, 12, 16])
        causal = rng.random() < 0.5
        return _sdpa("", "f32", rng.choice([1, 1, 2, 4]), h, h, s, s, rng.choice([64, 64, 80, 128]), causal,
                     "none" if causal else rng.choice(["none", "bool", "add"]), rng.choice(["bhsd", "bshd"]))
    if kind == "encoder":
        s, h = _log_int(rng, 32, 2048), rng.choice([8, 12, 16])
        return _sdpa("", half, rng.randint(1, 16), h, h, s, s, rng.choice([64, 64, 128]), False,
                     rng.choice(["none", "bool", "add"]), rng.choice(["bhsd", "bshd"]))
    if kind == "prefill":
        s = _log_int(rng, 64, 8192)
        return _sdpa("", half, rng.choice([1, 1, 2, 4]), hq, hkv, s, s, rng.choice([128, 128, 128, 64]), rng.random() < 0.85,
                     "none", rng.choice(["bhsd", "bshd"]))
    if kind == "cached":
        return _sdpa("", half, rng.choice([1, 2, 4, 8, 16]), hq, hkv, 1, _log_int(rng, 64, 8192), rng.choice([128, 128, 64]),
                     False, rng.choice(["none", "bool", "add"]), "cache")
    seed = rng.randint(1, 1 << 20)
    hi = _log_int(rng, 64, 32768 if kind == "decode" else 8192)
    lo = max(16, int(hi * rng.choice([0.06, 0.3, 1.0])))
    capacity = 1 << max(10, (hi + 1100).bit_length())
    if kind in ("decode", "decode16", "scores"):
        return _paged("", half, half if kind == "decode16" else "u8", hq, hkv, _log_int(rng, 1, 128), lo, hi,
                      capacity=capacity, lens_seed=seed, scores=kind == "scores")
    new_hi = _log_int(rng, 32, 1024)
    decode = 0 if kind == "chunks" else _log_int(rng, 4, 128)
    past_hi = rng.choice([0, 500, 4000])
    return _paged("", half, "u8", hq, hkv, decode, lo if decode else 0, hi if decode else 0, prefill=rng.randint(1, 8),
                  new_lo=max(2, int(new_hi * rng.choice([0.3, 1.0]))), new_hi=new_hi, past_hi=past_hi,
                  capacity=1 << max(10, (max(hi if decode else 0, past_hi + new_hi) + 1).bit_length()), lens_seed=seed)


def draw(rng):
    while True:
        case = _draw_once(rng)
        w = work(case)
        if w["flops"] <= MAX_FLOPS and w["bytes"] <= MAX_BYTES:
            return case


# ------------------------------------------------------------------------------------------------ lengths and work

def _lengths(case):
    """(past, new) tokens of every sequence of a paged case: prefill sequences first."""
    r = random.Random(case["lens_seed"])
    past, new = [], []
    for _ in range(case["prefill"]):
        new.append(r.randint(case["new_lo"], case["new_hi"]))
        past.append(r.randint(0, case["past_hi"]))
    for _ in range(case["decode"]):
        new.append(1)
        past.append(r.randint(case["ctx_lo"], case["ctx_hi"]) - 1)
    return past, new


def work(case):
    if case["family"] == "sdpa":
        es = 4 if case["dtype"] == "f32" else 2
        b, hq, hkv, sq, skv, d = (case[k] for k in ("b", "hq", "hkv", "sq", "skv", "d"))
        pairs = sq * (sq + 1) // 2 if case["causal"] else sq * skv
        return {"bytes": es * d * b * (2 * hq * sq + 2 * hkv * skv), "flops": 4 * b * hq * d * pairs}
    d = 128
    past, new = _lengths(case)
    tokens = sum(new)
    row = case["hkv"] * 2 * (d + 4 if case["kv"] == "u8" else 2 * d)  # K and V of one cached token
    cached = sum(p + n for p, n in zip(past, new))
    pairs = sum(n * p + n * (n + 1) // 2 for p, n in zip(past, new))
    step = tokens * (2 * 2 * case["hq"] * d + 2 * 2 * case["hkv"] * d)  # query, output, new K and V
    scores = cached * 4 if case["scores"] else 0
    return {"bytes": cached * row + tokens * row + step + scores, "flops": 4 * case["hq"] * d * pairs}


def tolerance(case):
    # About four times what is seen against a float64 restatement on the same inputs.  float32 (seen 3.3e-7): the order
    # of float32 sums.  16-bit (seen 4.2e-4 in f16, 2.1e-3 in bf16): the rounding of the result and of the probabilities
    # that enter the second product.  Long contexts (seen 1.7e-3 up to 8192 tokens, 6.7e-3 at 32768, f16): the average
    # of many values is small against the float32 sums over unscaled cache codes that it is the difference of.  The
    # cache bytes and the status word that a paged step returns stay the same.
    if case["dtype"] == "f32":
        return {"rel": 2e-6, "max": 3e-5}
    rel, most = (2e-3, 2.2e-2) if case["dtype"] == "f16" else (8.5e-3, 1.8e-1)
    if case["family"] == "paged":
        past, new = _lengths(case)
        rel = max(rel, min(2.7e-2, 1e-6 * max(p + n for p, n in zip(past, new))))
        most = max(most, 3 * rel)
    return {"rel": rel, "max": most}


# ------------------------------------------------------------------------------------------------------- the inputs

def _prepare_sdpa(case, gen):
    dt = DTYPES[case["dtype"]]
    b, hq, hkv, sq, skv, d = (case[k] for k in ("b", "hq", "hkv", "sq", "skv", "d"))

    def operand(h, s, rows):
        if case["layout"] == "bshd":
            return torch.randn(b, s, h, d, generator=gen, device="cuda").to(dt).transpose(1, 2)
        return torch.randn(b, h, rows, d, generator=gen, device="cuda").to(dt)[:, :, :s]
    kv_rows = (skv + 1023) // 1024 * 1024 if case["layout"] == "cache" else skv
    q, k, v = operand(hq, sq, sq), operand(hkv, skv, kv_rows), operand(hkv, skv, kv_rows)
    mask = None
    if case["mask"] != "none":
        lens = torch.randint((skv + 1) // 2, skv + 1, (b, 1), generator=gen, device="cuda")
        at = torch.arange(skv, device="cuda").expand(b, skv)
        keep = (at >= skv - lens if case["sq"] == 1 else at < lens).reshape(b, 1, 1, skv)  # left / right padding
        mask = keep if case["mask"] == "bool" else torch.where(keep, 0.0, torch.finfo(dt).min).to(dt)
    out = torch.empty(b, sq, hq, d, dtype=dt, device="cuda").transpose(1, 2) if case["layout"] == "bshd" \
        else torch.empty(b, hq, sq, d, dtype=dt, device="cuda")
    return {"family": "sdpa", "op": b2a.SdpaOp(causal=case["causal"]), "inputs": [q, k, v] + ([mask] if mask is not None else []),
            "out": out}


def _prepare_paged(case, seed, gen):
    dt, kv, hq, hkv, d = DTYPES[case["dtype"]], DTYPES[case["kv"]], case["hq"], case["hkv"], 128
    past, new = _lengths(case)
    n, tokens = len(past), sum(new)
    blocks = sum((p + m + BLOCK - 1) // BLOCK for p, m in zip(past, new)) + 8
    cache = b2a.PagedKvCache.allocate(blocks, hkv, d, BLOCK, kv)
    mgr = b2a.KvBlockManager(blocks, BLOCK, shuffle_seed=seed + 1)
    for s in range(n):
        mgr.add_sequence(s)
    rows = lambda t, h: torch.randn(t, h * d, generator=gen, device="cuda", dtype=dt)  # noqa: E731
    # what earlier steps have cached, a slice of every sequence at a time
    for at in range(0, max(past), 4096):
        ids = [s for s in range(n) if past[s] > at]
        tables = mgr.schedule_step(ids, [min(past[s] - at, 4096) for s in ids])
        t = [torch.from_numpy(x).cuda() for x in tables[:4]]
        b2a.paged_kv_store(rows(int(tables[1][-1]), hkv), rows(int(tables[1][-1]), hkv), cache, *t)
    tables = mgr.schedule_step(list(range(n)), new)
    op = b2a.PagedAttentionOp(hq, hkv, d, BLOCK, kv, max_seqs=n, max_context_len=case["capacity"], q_dtype=dt,
                              max_prefill_kv_tokens=mgr.last_prefill_kv_tokens, max_step_tokens=max(tokens, case["capacity"]))
    outputs = [torch.empty(tokens, hq * d, dtype=dt, device="cuda")]
    if case["scores"]:
        outputs.append(torch.zeros(sum(past) + tokens, dtype=torch.float32, device="cuda"))
    return {"family": "paged", "op": op, "cache": cache, "outputs": outputs,
            "inputs": [rows(tokens, hq), rows(tokens, hkv), rows(tokens, hkv), cache.k, cache.v,
                       *[torch.from_numpy(x).cuda() for x in tables[:4]], None, 0],
            "work": {"mutable": [torch.empty(m, dtype=torch.uint8, device="cuda") for m in op.GetWorkBufferRequest()["mutable_sizes"]]},
            "status": torch.zeros(1, dtype=torch.int32, device="cuda"),
            "hints": {"prefill_row_blocks": mgr.last_prefill_row_blocks, "prefill_kv_tokens": mgr.last_prefill_kv_tokens}}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["family"] == "sdpa":
        return _prepare_sdpa(case, gen)
    return _prepare_paged(case, seed, gen)


def run(state):
    if state["family"] == "sdpa":
        state["op"].Execute(state["inputs"], [state["out"]])
        return state["out"]
    begins = state["op"].Execute(state["inputs"], state["outputs"], workbuffers=state["work"], status=state["status"], **state["hints"])
    return {"outputs": state["outputs"], "score_begins": begins, "k_cache": state["cache"].k, "v_cache": state["cache"].v,
            "status": state["status"]}

"""The work this package is timed on: decode steps, quantize-pack and whole short generations.

Sizes are those of the benchmark's workloads and of the tests (batch 1 to 32, 32/8, 64/8 and 32/32 query/KV
heads of 128 dims, up to 128 Ki cached tokens, 4 and 2 bits, groups of 128, 64 and 32, fp16 and bf16), plus odd
and ragged ones of the same ranges.  Every case goes through the public entry points only.

A case is a dict of plain values:

* ``kind``: "step" a prepared ``DecodeStep`` (what a decoder loop keeps), "call" one ``fwd_kvcache_int`` call,
  "pack" one ``kvcache_pack_int`` call, "generate" a ``PackedKVCache`` that takes a batch of prompts and then
  ``tokens`` decoder steps with rotary embedding, appends and roll-overs;
* ``b, h, h_k, s``: sequences, query heads, KV heads, (longest) packed length or prompt length in tokens;
* ``bits, group, dtype``: the cache's format and the type of q, K and V;
* ``tail``: unquantized tokens behind the packed ones; ``ragged``: every sequence has lengths of its own;
  ``page``: tokens per page of a paged cache (0: contiguous); ``lse``: the log-sum-exp is asked for as well.
"""
import math

import torch

import bitladder_b200 as B
from bitladder_b200.kv_cache import PackedKVCache

D = 128
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _case(kind, b, h, h_k, s, bits, group, dtype, tail=0, ragged=False, page=0, lse=False, tokens=0):
    return dict(kind=kind, b=b, h=h, h_k=h_k, s=s, bits=bits, group=group, dtype=dtype, tail=tail, ragged=ragged,
                page=page, lse=lse, tokens=tokens)


def listed():
    return [
        # one user, a short context: the step is launch and dependency latency
        dict(_case("step", 1, 32, 8, 4096, 4, 128, "fp16"), name="step_b1_4k"),
        # the same length with a KV head per query head and the finest group, through the drop-in call
        dict(_case("call", 1, 32, 32, 4096, 4, 32, "fp16"), name="call_b1_mha_4k_g32"),
        # the benchmark's headline: a batch of eight 32 Ki contexts with a half-full tail
        dict(_case("step", 8, 32, 8, 32768, 4, 128, "fp16", tail=64), name="step_b8_32k_tail"),
        # one long document at the lowest precision
        dict(_case("call", 1, 32, 8, 131072, 2, 64, "fp16", lse=True), name="call_b1_128k_2bit"),
        # a serving batch of unequal contexts, multi-head attention, bf16
        dict(_case("call", 32, 32, 32, 16384, 4, 128, "bf16", tail=128, ragged=True), name="call_b32_ragged_mha"),
        # large batch times long context, eight query heads per KV head, at both precisions
        dict(_case("step", 16, 64, 8, 131072, 4, 128, "fp16"), name="step_b16_128k"),
        dict(_case("step", 16, 64, 8, 131072, 2, 128, "fp16"), name="step_b16_128k_2bit"),
        # a paged pool shared by requests of odd lengths
        dict(_case("call", 16, 32, 8, 8192, 4, 128, "bf16", tail=100, ragged=True, page=256), name="call_paged_b16_8k"),
        # the tails of a batch quantized as their next block (what a decoder does once per 128 tokens)
        dict(_case("pack", 8, 32, 8, 128, 4, 128, "fp16"), name="pack_block_b8"),
        # prompts quantized after prefill
        dict(_case("pack", 8, 32, 8, 32768, 4, 128, "fp16"), name="pack_b8_32k"),
        dict(_case("pack", 2, 32, 32, 16384, 2, 64, "bf16"), name="pack_b2_16k_mha_2bit"),
        # a whole short exchange: prompts of unequal lengths, then 48 tokens for each of them
        dict(_case("generate", 8, 32, 8, 2000, 4, 128, "fp16", ragged=True, tokens=48), name="generate_b8_2k"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["step", "step", "call", "call", "pack", "generate"])
    h, h_k = rng.choice([(32, 8), (32, 8), (64, 8), (32, 32), (16, 4), (8, 1), (16, 1)])
    bits = rng.choice([4, 4, 2])
    group = rng.choice([128, 128, 64, 32] if bits == 4 else [128, 64])
    dtype = rng.choice(["fp16", "bf16"])
    block = B.pack_block_tokens(bits)
    if kind == "generate":
        b = rng.randint(1, 12)
        return _case(kind, b, h, h_k, _log_int(rng, 100, 4000), bits, group, dtype, ragged=rng.random() < 0.6,
                     tokens=rng.randint(4, 48))
    b = _log_int(rng, 1, 32)
    # at most the packed tokens times heads of the largest listed case (a quarter of that for pack, which reads
    # the unquantized rows)
    most = (16 * 131072 * 8 if kind != "pack" else 8 * 32768 * 8) // (b * h_k)
    s = _log_int(rng, block, min(most, 1 << 18))
    if kind == "pack":
        return _case(kind, b, h, h_k, max(block, s // block * block), bits, group, dtype)
    page = rng.choice([0, 0, 0, 256, 512]) if kind == "call" else 0
    return _case(kind, b, h, h_k, s, bits, group, dtype, tail=rng.choice([0, 1, 17, 64, 100, 128]),
                 ragged=rng.random() < 0.5, page=page, lse=rng.random() < 0.25)


def _lengths(case):
    """(packed tokens, tail tokens) of every sequence; the same for every seed, so that a pass is the same work."""
    n, b, r = case["s"], case["b"], case["tail"]
    if not case["ragged"]:
        return [n] * b, [r] * b
    lo = max(1, n // 16)
    # evenly spread over [s/16, s], in a scattered order; the longest sequence has s tokens
    lens = [n - (n - lo) * ((7 * i) % b) // max(1, b - 1) if b > 1 else n for i in range(b)]
    if case["kind"] != "generate":
        block = B.pack_block_tokens(case["bits"])
        lens = [max(1, x // block * block) if r else x for x in lens]     # with a tail: whole blocks, as a cache holds them
    return lens, [max(0, r - (5 * i) % (r + 1)) for i in range(b)]


def _rows(gen, shape, dtype, k):
    """K or V rows: normal values; K with the few large channels that keys have, the same in every sequence."""
    x = torch.randn(shape, generator=gen, device="cuda", dtype=dtype)
    if k:
        x[..., 5::31] *= 4
    return x


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, b, h, h_k, s = case["kind"], case["b"], case["h"], case["h_k"], case["s"]
    bits, group, dtype = case["bits"], case["group"], DTYPES[case["dtype"]]
    block = B.pack_block_tokens(bits)
    scale = 1.0 / math.sqrt(D)
    fmt = ("k-channel", group, bits)
    if kind == "pack":
        k, v = (_rows(gen, (b, s, h_k, D), dtype, x) for x in (True, False))
        return dict(kind=kind, k=k, v=v, s=s, fmt=fmt, bufs=B.alloc_packed_cache(b, s, h_k, D, bits, group))
    if kind == "generate":
        n = case["tokens"]
        k, v = (_rows(gen, (b, s, h_k, D), dtype, x) for x in (True, False))
        q = torch.randn(n, b, 1, h, D, generator=gen, device="cuda", dtype=dtype)
        kn, vn = (_rows(gen, (n, b, 1, h_k, D), dtype, x) for x in (True, False))
        angle = torch.arange(s + n, device="cuda")[:, None] * 10000.0 ** (-torch.arange(D // 2, device="cuda") / (D // 2))
        cache = PackedKVCache(b, s + n + block, h_k, D, bits, group, dtype)
        return dict(kind=kind, cache=cache, k=k, v=v, q=q, kn=kn, vn=vn, scale=scale, lens=_lengths(case)[0],
                    cos=angle.cos().to(dtype), sin=angle.sin().to(dtype))
    # a packed cache, filled sequence by sequence (page by page where it is paged)
    lens, tails = _lengths(case)
    page = case["page"]
    table = None
    if page:
        per = (s + page - 1) // page
        pages = b * per
        order = torch.randperm(pages, generator=gen, device="cuda").to(torch.int32)
        table = order.view(b, per)
        rows = [page] * pages
    else:
        rows = [max(block, (s + block - 1) // block * block)] * b
    bufs = B.alloc_packed_cache(len(rows), rows[0], h_k, D, bits, group)
    step = max(1, (1 << 20) // rows[0])
    for i in range(0, len(rows), step):
        j = min(len(rows), i + step)
        k, v = (_rows(gen, (j - i, rows[0], h_k, D), dtype, x) for x in (True, False))
        B.kvcache_pack_int(k, bufs[0][i:j], bufs[1][i:j], v, bufs[2][i:j], bufs[3][i:j], None, None, rows[0], *fmt)
    q = torch.randn(b, 1, h, D, generator=gen, device="cuda", dtype=dtype)
    kw = {}
    if case["tail"]:
        kw["k_res"], kw["v_res"] = (_rows(gen, (b, case["tail"], h_k, D), dtype, x) for x in (True, False))
    if case["ragged"]:
        kw["cache_seqlens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
        if case["tail"]:
            kw["res_lens"] = torch.tensor(tails, dtype=torch.int32, device="cuda")
    args = (q, *bufs, table, scale, *fmt)
    kw.update(seqlen_k=s, return_lse=case["lse"])
    if kind == "step":
        return dict(kind=kind, step=B.DecodeStep(*args, **kw))
    return dict(kind=kind, args=args, kw=kw)


def run(state):
    kind = state["kind"]
    if kind == "step":
        return state["step"].step()
    if kind == "call":
        return B.fwd_kvcache_int(*state["args"], **state["kw"])
    if kind == "pack":
        k_pack, k_params, v_pack, v_params = state["bufs"]
        B.kvcache_pack_int(state["k"], k_pack, k_params, state["v"], v_pack, v_params, None, None, state["s"],
                           *state["fmt"])
        return [x.view(torch.int16) for x in state["bufs"]]      # codes, and pairs of fp16 scale and zero, bit for bit
    cache = state["cache"]
    cache.prefill(state["k"], state["v"], state["lens"])
    outs = [cache.append_and_decode(q, kn, vn, state["scale"], rotary_cos=state["cos"], rotary_sin=state["sin"])
            for q, kn, vn in zip(state["q"], state["kn"], state["vn"])]
    packed = [x.view(torch.int16) for x in (cache.k_pack, cache.k_params, cache.v_pack, cache.v_params)]
    return outs, packed, cache.k_tail, cache.v_tail, cache.cache_seqlens, cache.res_lens


def _packed_bytes(tokens, case):
    per_token = 2 * D * case["bits"] // 8 + D * 4 // case["group"] + D // case["group"] * 4
    return tokens * case["h_k"] * per_token


def work(case):
    lens, tails = _lengths(case)
    b, h, h_k = case["b"], case["h"], case["h_k"]
    row = 2 * h_k * D * 2                              # K and V of one unquantized token
    qo = 2 * b * h * D * 2
    if case["kind"] == "pack":
        tokens = b * case["s"]
        return {"bytes": tokens * row + _packed_bytes(tokens, case), "flops": 0}
    if case["kind"] != "generate":
        return {"bytes": _packed_bytes(sum(lens), case) + sum(tails) * row + qo, "flops": 4 * h * D * (sum(lens) + sum(tails))}
    block = B.pack_block_tokens(case["bits"])
    total = {"bytes": 0, "flops": 0}
    for n in lens:
        full = n // block * block
        total["bytes"] += n * row + _packed_bytes(full, case) + (n - full) * row
        for i in range(case["tokens"]):
            full, tail = (n + i) // block * block, (n + i) % block
            total["bytes"] += _packed_bytes(full, case) + (tail + 2) * row + qo // b
            total["flops"] += 4 * h * D * (n + i + 1)
            if tail + 1 == block:
                total["bytes"] += block * row + _packed_bytes(block, case)
    return total


def tolerance(case):
    if case["kind"] == "pack":
        return "exact"                                 # bytes of a defined format
    # Four times and more what separates the kernels from an evaluation in 64 bits of the same codes and tails (two
    # sequences of 256 to 32768 tokens, both bit widths, groups 64 and 128): fp16 at most 1.6e-3 and 1.2e-2, growing with
    # the length as the average over V shrinks (probabilities and their products with the scales are rounded to
    # fp16); bf16, whose output is rounded to 8 bits, at most 2.4e-3 and 1.2e-2.
    return {"rel": 8e-3, "max": 6e-2} if case["dtype"] == "fp16" else {"rel": 1.2e-2, "max": 8e-2}

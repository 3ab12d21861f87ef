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
    """K or V rows: normal values; K with the few large channels that keys have, V about a mean of every channel that its
    tokens share (so that the average over a long context does not vanish), the same in every sequence."""
    x = torch.randn(shape, generator=gen, device="cuda", dtype=dtype)
    if k:
        x[..., 5::31] *= 4
    else:
        x += torch.linspace(-1, 1, D, device="cuda", dtype=dtype)
    return x


def _cached_rows(gen, case):
    """Where the cache's blocks go (page table or None, and the rows of every sequence or page), then its unquantized rows
    in the order they are packed, as (first, last, k, v)."""
    b, s, page, block = case["b"], case["s"], case["page"], B.pack_block_tokens(case["bits"])
    table, n, rows = None, b, max(block, (s + block - 1) // block * block)
    if page:
        per = (s + page - 1) // page
        n, rows = b * per, page
        table = torch.randperm(n, generator=gen, device="cuda").to(torch.int32).view(b, per)
    yield table, n, rows
    step = max(1, (1 << 20) // rows)
    for i in range(0, n, step):
        j = min(n, i + step)
        k, v = (_rows(gen, (j - i, rows, case["h_k"], D), DTYPES[case["dtype"]], x) for x in (True, False))
        yield i, j, k, v


def _query_and_tail(gen, case):
    b, dtype, tail = case["b"], DTYPES[case["dtype"]], case["tail"]
    q = torch.randn(b, 1, case["h"], D, generator=gen, device="cuda", dtype=dtype)
    return q, [_rows(gen, (b, tail, case["h_k"], D), dtype, x) for x in (True, False)] if tail else None


def _exchange(gen, case):
    """A generation's prompts, its tokens' queries and rows, and the rotary tables."""
    b, s, n, h_k, dtype = case["b"], case["s"], case["tokens"], case["h_k"], DTYPES[case["dtype"]]
    k, v = (_rows(gen, (b, s, h_k, D), dtype, x) for x in (True, False))
    q = torch.randn(n, b, 1, case["h"], D, generator=gen, device="cuda", dtype=dtype)
    kn, vn = (_rows(gen, (n, b, 1, h_k, D), dtype, x) for x in (True, False))
    angle = torch.arange(s + n, device="cuda")[:, None] * 10000.0 ** (-torch.arange(D // 2, device="cuda") / (D // 2))
    return dict(k=k, v=v, q=q, kn=kn, vn=vn, cos=angle.cos().to(dtype), sin=angle.sin().to(dtype))


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
        cache = PackedKVCache(b, s + case["tokens"] + block, h_k, D, bits, group, dtype)
        return dict(kind=kind, cache=cache, scale=scale, lens=_lengths(case)[0], **_exchange(gen, case))
    # a packed cache, filled sequence by sequence (page by page where it is paged)
    lens, tails = _lengths(case)
    rows = _cached_rows(gen, case)
    table, n, per = next(rows)
    bufs = B.alloc_packed_cache(n, per, h_k, D, bits, group)
    for i, j, k, v in rows:
        B.kvcache_pack_int(k, bufs[0][i:j], bufs[1][i:j], v, bufs[2][i:j], bufs[3][i:j], None, None, per, *fmt)
    q, tail = _query_and_tail(gen, case)
    kw = {}
    if tail:
        kw["k_res"], kw["v_res"] = tail
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


def _dequantized(x, dim, case):
    """(tokens, KV heads, D) rows as the cache's codes, scales and zeros hold them (groups along `dim`), in 64 bits."""
    bits, group = case["bits"], case["group"]
    x = x.float().unflatten(dim, (-1, group))
    dim = dim % 3 + 1
    lo, hi = x.amin(dim, keepdim=True), x.amax(dim, keepdim=True)
    top = torch.full_like(lo, 2 ** bits - 1)
    inv = torch.where(hi > lo, torch.div(top, hi - lo), 0 * top)
    scale = torch.where(inv == 0, 0 * top, torch.div(torch.ones_like(top), inv))
    codes = ((x - lo) * inv).add(0.5).floor().clamp(0, 2 ** bits - 1).double()
    return (codes * scale.half().double() + lo.half().double()).flatten(dim - 1, dim)


def _attend(q, k, v, scale):
    """(h, D) over (tokens, h_k, D): the output and the log-sum-exp of the scaled scores."""
    h_k = k.shape[1]
    scores = torch.einsum("hgd,thd->hgt", q.double().view(h_k, -1, D), k.double()) * scale
    lse = scores.logsumexp(-1)
    return torch.einsum("hgt,thd->hgd", (scores - lse[..., None]).exp(), v.double()).reshape(-1, D), lse.reshape(-1)


def _rotated(x, cos, sin):
    """(heads, D) at one position, pairs (2i, 2i + 1), in 64 bits."""
    a, b, cos, sin = x[..., ::2].double(), x[..., 1::2].double(), cos.double(), sin.double()
    return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(-2)


def exact(case, seed):
    if case["kind"] == "pack":
        return None                                    # bytes, not computed numbers
    gen = torch.Generator(device="cuda").manual_seed(seed)
    scale, block, dtype = 1.0 / math.sqrt(D), B.pack_block_tokens(case["bits"]), DTYPES[case["dtype"]]
    lens, tails = _lengths(case)
    if case["kind"] == "generate":
        x = _exchange(gen, case)
        outs = [torch.empty(case["b"], 1, case["h"], D, dtype=torch.float64, device="cuda") for _ in range(case["tokens"])]
        for i, n in enumerate(lens):
            full = n // block * block
            old = [_dequantized(x["k"][i, :full], 0, case), _dequantized(x["v"][i, :full], -1, case)] if full else \
                [torch.empty(0, case["h_k"], D, dtype=torch.float64, device="cuda")] * 2
            new = [x["k"][i, full:n], x["v"][i, full:n]]
            for t, out in enumerate(outs):
                cos, sin = x["cos"][n + t], x["sin"][n + t]
                new = [torch.cat([new[0], _rotated(x["kn"][t, i], cos, sin).to(dtype)]), torch.cat([new[1], x["vn"][t, i]])]
                out[i, 0] = _attend(_rotated(x["q"][t, i, 0], cos, sin), torch.cat([old[0], new[0].double()]),
                                    torch.cat([old[1], new[1].double()]), scale)[0]
                if len(new[0]) == block:
                    old = [torch.cat([o, _dequantized(y, dim, case)]) for o, y, dim in zip(old, new, (0, -1))]
                    new = [y[:0] for y in new]
        return outs, [None] * 4, None, None, None, None
    rows = _cached_rows(gen, case)
    table, n, per = next(rows)
    k, v = (torch.cat(x) for x in zip(*(r[2:] for r in rows)))
    q, tail = _query_and_tail(gen, case)
    out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    lse = torch.empty(q.shape[0], q.shape[2], dtype=torch.float64, device="cuda")
    for i, (n, r) in enumerate(zip(lens, tails)):
        whole = (n + block - 1) // block * block
        ki, vi = (x[table[i].long()].flatten(0, 1) if case["page"] else x[i] for x in (k, v))
        ki, vi = _dequantized(ki[:whole], 0, case)[:n], _dequantized(vi[:whole], -1, case)[:n]
        if r:
            ki, vi = torch.cat([ki, tail[0][i, :r].double()]), torch.cat([vi, tail[1][i, :r].double()])
        out[i, 0], lse[i] = _attend(q[i, 0], ki, vi, scale)
    return (out, lse) if case["lse"] else out

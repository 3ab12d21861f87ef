"""GPU: the kernel for steps with little work (a cluster of CTAs per sequence and KV head) against the oracle and against the
general kernel on the same inputs (`num_splits` > 0 asks for that one)."""
import numpy as np
import pytest
import torch

from tests import gpu_util as G, helpers as H

pytestmark = pytest.mark.gpu

FMT = lambda group, bits: ("k-channel", group, bits)


def _both(B, x, bufs, group, bits, table=None, **kw):
    """(out, lse) of the short kernel, checked against the general kernel's."""
    args = (x["q"].cuda(), *bufs, table, H.default_scale(), *FMT(group, bits))
    step = B.DecodeStep(*args, return_lse=True, **kw)
    assert step.plan()["warps_per_cta"] == 8 and step.plan()["launches"] == 1
    out, lse = step.step(check=True)
    o2, l2 = B.fwd_kvcache_int(*args, return_lse=True, num_splits=2, check=True, **kw)
    # The path's own bounds: q * scale and p * scale are rounded to fp16 in both, in another order of sums; with bf16 the
    # query, tail and output have 8 bits (the bounds are 8 times the fp16 ones).
    dtype = "fp16" if x["q"].dtype == torch.float16 else "bf16"
    assert (out.float() - o2.float()).abs().max() <= G.TOL_O[dtype] * max(1.0, float(o2.float().abs().max()))
    inf = torch.isinf(l2)
    assert torch.equal(torch.isinf(lse), inf) and ((lse - l2)[~inf].abs() <= G.TOL_LSE[dtype]).all()
    return out, lse


# (sequences, query heads, KV heads): clusters of 8, 4, 2 and 1 CTAs, and two CTAs in turn on an SM; one and two query tiles
@pytest.mark.parametrize("b,h,h_k", [(1, 8, 8), (1, 4, 1), (4, 64, 8), (5, 18, 2), (9, 32, 8), (17, 8, 8), (24, 8, 8), (3, 16, 1)])
@pytest.mark.parametrize("bits,group", [(4, 128), (4, 64), (4, 32), (2, 128), (2, 64), (2, 32)])
def test_against_oracle_and_general_kernel(b, h, h_k, bits, group):
    import bitladder_b200 as B
    if bits == 2 and group == 32 and h > 8 * h_k:
        pytest.skip("not built")
    block = B.pack_block_tokens(bits)
    dtype = "bf16" if (b + group) % 3 == 0 else "fp16"
    s = 4 * block
    x = H.gen_qkv(b, s, h, h_k, seed=b + group, dtype=dtype, res=40)
    bufs = G.pack_gpu(B, x["k"], x["v"], bits, group)
    # lengths at the edges of half blocks, blocks and tail items, empty ones among them
    lens = torch.tensor([[0, 1, 16, 31, 32, block - 1, block, block + 1, block + 17, 3 * block, s - 1, s][i * 5 % 12] for i in range(b)],
                        dtype=torch.int32)
    tails = torch.tensor([[0, 1, 15, 16, 17, 40][i % 6] for i in range(b)], dtype=torch.int32)
    kw = dict(cache_seqlens=lens.cuda(), res_lens=tails.cuda(), k_res=x["k_res"].cuda(), v_res=x["v_res"].cuda())
    out, lse = _both(B, x, bufs, group, bits, **kw)
    ref = H.oracle_pack(x["k"], x["v"], bits, group, dtype)
    o_ref, l_ref = H.oracle_decode(x["q"], ref, H.default_scale(), bits, group, dtype, k_res=x["k_res"], v_res=x["v_res"],
                                   res_lens=tails.numpy(), cache_seqlens=lens.numpy())
    eo, el = G.errs(out, lse, o_ref, l_ref)
    assert eo <= G.TOL_O[dtype] and el <= G.TOL_LSE[dtype]


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("s", [1, 128, 1000, 4096])
def test_equal_lengths_strided_query_and_32_bit_output(bits, s):
    import bitladder_b200 as B
    cap = (s + 255) // 256 * 256
    x = H.gen_qkv(3, cap, 12, 4, seed=s)
    bufs = G.pack_gpu(B, x["k"], x["v"], bits, 128)
    wide = torch.zeros(3, 1, 24, 128, dtype=torch.float16, device="cuda")
    wide[:, :, ::2] = x["q"].cuda()
    args = (*bufs, None, H.default_scale(), *FMT(128, bits))
    got = B.fwd_kvcache_int(wide[:, :, ::2], *args, seqlen_k=s, out_dtype=torch.float32)
    want = B.fwd_kvcache_int(x["q"].cuda(), *args, seqlen_k=s, out_dtype=torch.float32, num_splits=1)
    assert got.dtype == torch.float32 and (got - want).abs().max() <= 2e-3


@pytest.mark.parametrize("bits", [4, 2])
def test_pages_in_any_order_and_one_outside_the_pool(bits):
    import bitladder_b200 as B
    from bitladder_b200 import _lib
    b, h, h_k, page, per = 3, 8, 2, 256, 4
    x = H.gen_qkv(b, page * per, h, h_k, seed=5)
    table = torch.randperm(b * per, generator=torch.Generator().manual_seed(3)).to(torch.int32).view(b, per)
    pool = [torch.empty(b * per, page, h_k, 128, dtype=torch.float16) for _ in range(2)]
    for p, t in zip(pool, (x["k"], x["v"])):
        p[table.flatten().long()] = t.reshape(b * per, page, h_k, 128)
    bufs = G.pack_gpu(B, *pool, bits, 128)
    lens = torch.tensor([page * per, 300, 700], dtype=torch.int32)
    out, lse = _both(B, x, bufs, 128, bits, table=table.cuda(), cache_seqlens=lens.cuda())
    ref = H.oracle_pack(x["k"], x["v"], bits, 128, "fp16")
    o_ref, l_ref = H.oracle_decode(x["q"], ref, H.default_scale(), bits, 128, "fp16", cache_seqlens=lens.numpy())
    eo, el = G.errs(out, lse, o_ref, l_ref)
    assert eo <= 2e-3 and el <= 2e-3
    table[0, per - 1] = b * per + 7
    step = B.DecodeStep(x["q"].cuda(), *bufs, table.cuda(), H.default_scale(), *FMT(128, bits), cache_seqlens=lens.cuda())
    out = step.step()
    assert step.status() == _lib.BD_ERR_PAGE
    lens[0] = page * (per - 1)
    o_ref, _ = H.oracle_decode(x["q"], ref, H.default_scale(), bits, 128, "fp16", cache_seqlens=lens.numpy())
    assert np.abs(out[:, 0].float().cpu().numpy() - o_ref).max() <= 2e-3


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("rotary_dim,interleaved", [(128, True), (128, False), (64, False), (48, True), (32, False), (16, False)])
def test_rotation_while_loading_files_the_same_key(dtype, rotary_dim, interleaved):
    """Tables that do not start on 16 bytes take the rotary kernel in front: the same bits in the tail, and the same output up
    to nothing at all, as the rotated query is the same too."""
    import bitladder_b200 as B
    x = H.gen_qkv(3, 512, 8, 2, seed=rotary_dim, dtype=dtype, res=64)
    bufs = G.pack_gpu(B, x["k"], x["v"], 4, 128)
    g = torch.Generator().manual_seed(1)
    tdt = torch.float16 if dtype == "fp16" else torch.bfloat16
    flat = [torch.randn(700 * rotary_dim // 2 + 8, generator=g).to(tdt).cuda() for _ in range(2)]
    new = [torch.randn(3, 1, 2, 128, generator=g).to(tdt).cuda() for _ in range(2)]
    got = []
    for off in (0, 1):
        tabs = [torch.empty(700 * rotary_dim // 2 + 8, dtype=tdt, device="cuda")[off:off + 700 * rotary_dim // 2] for _ in range(2)]
        for t, f in zip(tabs, flat):
            t.copy_(f[:t.numel()])
        tail = [x["k_res"].cuda().clone(), x["v_res"].cuda().clone()]
        step = B.DecodeStep(x["q"].cuda(), *bufs, None, H.default_scale(), *FMT(128, 4), return_lse=True, k_res=tail[0], v_res=tail[1],
                            cache_seqlens=torch.tensor([512, 100, 0], dtype=torch.int32, device="cuda"),
                            res_lens=torch.tensor([0, 17, 63], dtype=torch.int32, device="cuda"), k_new=new[0], v_new=new[1],
                            rotary_cos=tabs[0].view(700, -1), rotary_sin=tabs[1].view(700, -1), rotary_interleaved=interleaved)
        assert step.plan()["launches"] == 1 + off
        out, lse = step.step(check=True)
        got.append([out.clone(), lse.clone(), *tail])
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("bits,group,dtype,h,h_k", [(4, 128, "fp16", 8, 2), (4, 64, "bf16", 16, 16), (4, 32, "fp16", 18, 2), (2, 128, "bf16", 8, 8),
                                                    (2, 64, "fp16", 4, 1), (2, 32, "fp16", 8, 2)])
def test_roll_over_leaves_the_same_bytes_as_the_general_kernels(bits, group, dtype, h, h_k):
    """A step with bookkeeping: tails that are not full, that this step fills, that fill with no room behind them, and a full
    one; lengths, tails, packed bytes and the reported error are those of the general kernel and the roll-over kernel."""
    import bitladder_b200 as B
    block = B.pack_block_tokens(bits)
    cap = 3 * block
    tdt = torch.float16 if dtype == "fp16" else torch.bfloat16
    x = H.gen_qkv(5, cap, h, h_k, seed=bits + group, dtype=dtype, res=block)
    x["k_res"][:, ::7, :, 3] = 1e-39 if dtype == "bf16" else 6e-8       # subnormal rows are not flushed
    g = torch.Generator().manual_seed(2)
    new = [torch.randn(5, 1, h_k, 128, generator=g).to(tdt).cuda() for _ in range(2)]
    got = []
    for splits in (0, 2):
        bufs = [t.clone() for t in G.pack_gpu(B, x["k"], x["v"], bits, group)]
        tail = [x["k_res"].cuda().clone(), x["v_res"].cuda().clone()]
        cs = torch.tensor([block, 0, 2 * block, cap, block], dtype=torch.int32, device="cuda")
        rl = torch.tensor([block - 1, block - 1, block - 2, block - 1, block], dtype=torch.int32, device="cuda")
        step = B.DecodeStep(x["q"].cuda(), *bufs, None, H.default_scale(), *FMT(group, bits), return_lse=True, k_res=tail[0], v_res=tail[1],
                            cache_seqlens=cs, res_lens=rl, k_new=new[0], v_new=new[1], advance=True, num_splits=splits)
        if splits == 0:
            assert step.plan()["launches"] == 1
        out, lse = step.step()
        got.append(([t.view(torch.int16) for t in (*bufs, *tail)] + [cs, rl], out.float(), lse, step.status()))
    (a, oa, la, sa), (b, ob, lb, sb) = got
    assert all(torch.equal(s, t) for s, t in zip(a, b)) and sa == sb != 0
    assert a[6].tolist() == [2 * block, block, 2 * block, cap, 2 * block] and a[7].tolist() == [0, 0, block - 1, block, 0]
    # a tail that was full from the start is packed as it is
    want = [t.clone() for t in G.pack_gpu(B, x["k"], x["v"], bits, group)]
    rows = [x[n][4:].cuda() for n in ("k_res", "v_res")]
    B.kvcache_pack_int(rows[0], want[0][4:], want[1][4:], rows[1], want[2][4:], want[3][4:], None, None, block, *FMT(group, bits),
                       dst_token_offset=block)
    assert all(torch.equal(s[4], t.view(torch.int16)[4]) for s, t in zip(a, want))
    assert (oa - ob).abs().max() <= G.TOL_O[dtype] * max(1.0, float(ob.abs().max())) and (la - lb).abs().max() <= G.TOL_LSE[dtype]


def _cluster(B, b, h, h_k, s, bits, group, tail=0, ragged=False, advance=False):
    """CTAs per (sequence, KV head) of the short kernel that the step would run; 0: the general kernel."""
    i32 = lambda n: torch.full((b,), n, dtype=torch.int32, device="cuda")
    rows = lambda n, heads: torch.zeros(b, n, heads, 128, dtype=torch.float16, device="cuda")
    block = B.pack_block_tokens(bits)
    kw = dict(k_res=rows(tail, h_k), v_res=rows(tail, h_k)) if tail else {}
    if ragged:
        kw["cache_seqlens"] = i32(block)
        if tail:
            kw["res_lens"] = i32(1)
    if advance:
        kw.update(k_new=rows(1, h_k), v_new=rows(1, h_k), advance=True)
    bufs = B.alloc_packed_cache(b, (s + block - 1) // block * block, h_k, 128, bits, group)
    plan = B.DecodeStep(rows(1, h), *bufs, None, 0.1, *FMT(group, bits), seqlen_k=s, **kw).plan()
    c = plan["rows"] // b
    return c if plan["warps_per_cta"] == 8 and plan["launches"] == 1 and plan["rows"] == b * c and c in (1, 2, 4, 8) else 0


@pytest.mark.parametrize("pairs,most", [(15, 8), (16, 4), (17, 4), (33, 4), (34, 2), (37, 2), (74, 2), (75, 1)])
def test_clusters_are_no_larger_than_run_at_once(pairs, most):
    """On a B200 15 clusters of 8 CTAs, 33 of 4 and 74 of 2; the results with those sizes are the general kernel's."""
    import bitladder_b200 as B
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes of a device with 148 SMs")
    assert _cluster(B, pairs, 4, 1, most * 1024, 4, 128, ragged=True) == most          # two rounds
    x = H.gen_qkv(pairs, 512, 4, 1, seed=pairs)
    lens = (torch.arange(pairs, dtype=torch.int32) * 97 % 513).cuda()
    _both(B, x, G.pack_gpu(B, x["k"], x["v"], 4, 128), 128, 4, cache_seqlens=lens)


# (sequences, query heads, KV heads, tokens, bits, group, tail, lengths per sequence): on either side of the rule's limits, which
# lie lower where the clusters take few SMs and a round is long
@pytest.mark.parametrize("little,shape", [
    (True, (1, 32, 8, 4096, 4, 128, 0, False)), (True, (8, 32, 8, 2048, 4, 128, 128, True)), (True, (8, 32, 32, 2000, 2, 64, 64, True)),
    (True, (1, 16, 1, 4096, 2, 64, 0, False)), (False, (1, 16, 1, 12288, 2, 64, 0, False)),
    (False, (4, 64, 4, 24320, 4, 128, 64, False)), (False, (2, 32, 8, 49152, 2, 128, 0, False)),
    (True, (1, 32, 8, 8192, 2, 64, 0, False)), (False, (1, 32, 8, 16384, 2, 64, 0, False)),
    (True, (1, 32, 8, 5888, 4, 32, 64, True)), (False, (1, 32, 8, 7936, 4, 32, 64, True)),
    (True, (2, 32, 8, 1024, 4, 128, 0, True)), (True, (3, 32, 32, 1536, 4, 32, 0, True)), (False, (3, 32, 32, 2048, 4, 32, 0, True)), (False, (4, 32, 32, 4096, 2, 128, 0, True)),
    (True, (8, 32, 32, 1024, 4, 128, 64, True)), (False, (8, 32, 32, 1536, 4, 32, 0, False)), (False, (20, 32, 8, 2048, 4, 128, 64, False)),
    (True, (15, 32, 8, 2048, 4, 32, 0, True)), (True, (32, 32, 8, 2048, 4, 128, 0, False)), (False, (32, 32, 8, 4096, 4, 128, 0, False)),
    (False, (36, 32, 8, 2048, 4, 128, 0, False)), (False, (32, 32, 8, 1024, 4, 32, 0, False))])
def test_which_steps_are_little_work(little, shape):
    import bitladder_b200 as B
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("limits of a device with 148 SMs")
    b, h, h_k, s, bits, group, tail, ragged = shape
    assert (_cluster(B, b, h, h_k, s, bits, group, tail, ragged) > 0) == little

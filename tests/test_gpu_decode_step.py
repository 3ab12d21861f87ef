"""`DecodeStep`: the prepared step must do exactly what `fwd_kvcache_int` does, call after call,
while the contents of its tensors change."""
import math

import pytest
import torch

from tests import gpu_util as G, helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [0, 2])
def test_prepared_step_equals_the_plain_call_and_follows_content_changes(splits):
    import bitladder_b200 as B
    x = H.gen_qkv(3, 2048, 32, 8, seed=17, res=32)
    bufs = G.pack_gpu(B, x["k"], x["v"], 4, 128)
    q = x["q"].cuda()
    k_res, v_res = x["k_res"].cuda(), x["v_res"].cuda()
    res_lens = torch.tensor([32, 7, 0], dtype=torch.int32, device="cuda")
    lens = torch.tensor([2048, 1000, 128], dtype=torch.int32, device="cuda")
    scale = 1.0 / math.sqrt(128)
    run = B.DecodeStep(q, *bufs, None, scale, "k-channel", 128, 4, k_res=k_res, v_res=v_res, res_lens=res_lens,
                       cache_seqlens=lens, return_lse=True, num_splits=splits)
    for it in range(3):
        o_ref, l_ref = B.fwd_kvcache_int(q, *bufs, None, scale, "k-channel", 128, 4, k_res=k_res, v_res=v_res,
                                         res_lens=res_lens, cache_seqlens=lens, return_lse=True, num_splits=splits)
        o, l = run.step()
        assert torch.equal(o, o_ref) and torch.equal(l, l_ref)
        # new contents in the same buffers: the prepared step must see them
        q.copy_(torch.randn_like(q))
        res_lens.copy_(torch.tensor([5 + it, 32, 1], dtype=torch.int32))
        lens.copy_(torch.tensor([1024, 2048 - 128 * it, 0], dtype=torch.int32))


@pytest.mark.parametrize("b,s,rotary,splits", [(1, 512, False, 0), (2, 256, True, 0), (3, 16384, False, 0), (1, 512, False, 8),
                                               (2, 256, True, 2)])
def test_captured_behind_copies_and_joined_streams(b, s, rotary, splits):
    """The step's first kernel may be staged early behind what runs in front of it: in a graph that is a copy of the
    query, or the join of a side stream that writes it; in a stream, a kernel that has just written it."""
    import bitladder_b200 as B
    x = {k: v.cuda() for k, v in H.gen_qkv(b, s, 8, 2, seed=3, res=128).items() if isinstance(v, torch.Tensor)}
    bufs = B.alloc_packed_cache(b, s, 2, 128, 4, 128)
    B.kvcache_pack_int(x["k"], bufs[0], bufs[1], x["v"], bufs[2], bufs[3], None, None, s, "k-channel", 128, 4)
    q, kw = torch.zeros_like(x["q"]), {}
    if rotary:
        a = torch.arange(s + 128, device="cuda")[:, None] * torch.linspace(1, 0.01, 64, device="cuda")
        kw = dict(k_res=x["k_res"], v_res=x["v_res"], k_new=x["k"][:, :1], v_new=x["v"][:, :1], rotary_cos=a.cos().half(),
                  rotary_sin=a.sin().half(), cache_seqlens=torch.full((b,), s, dtype=torch.int32, device="cuda"),
                  res_lens=torch.full((b,), 5, dtype=torch.int32, device="cuda"))
    step = B.DecodeStep(q, *bufs, None, H.default_scale(), "k-channel", 128, 4, num_splits=splits, **kw)
    q.copy_(x["q"])
    torch.cuda.synchronize()
    want = step.step().clone()
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(main):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            q.copy_(x["q"])                          # a copy node
            first = step.step().clone()
            side.wait_stream(main)
            with torch.cuda.stream(side):
                q.mul_(-1)
                q.mul_(-1)
            first.add_(0)
            main.wait_stream(side)                   # two nodes in front
            second = step.step().clone()
        for _ in range(3):
            q.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(first, want) and torch.equal(second, want)
    for _ in range(20):                              # stream launches behind the kernels that write the query
        q.zero_()
        q.add_(x["q"])
        out = step.step().clone()
        assert torch.equal(out, want)

"""The extension that takes plainly valid calls to the library: the same results as the Python path in every form of a
call, and whatever it does not take comes back to the Python path."""
import ctypes as C
import subprocess
import threading
import time

import pytest
import torch

from tests import helpers as H

SCALE = H.default_scale()


def test_calls_that_are_not_plainly_valid_come_back():
    """No CUDA tensor, a wrong number or kind of arguments: None, never an error (the Python code decides)."""
    from bitladder_b200 import _torch_calls as T, _lib, bit_decode_interface as I
    lib = _lib.load()
    T.bind(*(I.C.cast(f, I.C.c_void_p).value for f in (lib.bd_decode, lib.bd_pack, lib.bd_decode_workspace_bytes)))
    q = torch.zeros(1, 1, 8, 128, dtype=torch.float16)
    assert T.decode() is None and T.pack(q) is None
    assert T.decode({}, *[q] * 24) is None and T.pack(*[q] * 11) is None
    assert T.decode({}, *["x", 1, None, object(), 2.0, {}] * 4) is None


def _forms():
    """(keyword arguments of a call, head counts, bits, group, dtype); lengths of 2 sequences, up to 512 tokens."""
    for bits, group, dtype in [(4, 128, "fp16"), (2, 64, "bf16"), (4, 32, "bf16")]:
        yield from ((f, bits, group, dtype) for f in ("plain", "lse", "tail", "ragged", "append", "rotary", "out32", "splits",
                                                      "bound", "paged", "strided_q", "int_scale"))


@pytest.mark.gpu
@pytest.mark.parametrize("form,bits,group,dtype", list(_forms()))
def test_same_bits_as_the_python_path(form, bits, group, dtype, monkeypatch):
    import bitladder_b200 as B
    from bitladder_b200 import bit_decode_interface as I
    x = {k: v.cuda() for k, v in H.gen_qkv(2, 512, 8, 2, seed=5, dtype=dtype, res=256).items() if isinstance(v, torch.Tensor)}
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")

    def outputs():
        bufs = B.alloc_packed_cache(2, 512, 2, 128, bits, group)
        B.kvcache_pack_int(x["k"], bufs[0], bufs[1], x["v"], bufs[2], bufs[3], None, None, 512, "k-channel", group, bits)
        q, table, scale, kw = x["q"], None, SCALE, {}
        k_res, v_res = x["k_res"].clone(), x["v_res"].clone()
        lens = dict(cache_seqlens=i32(512, 256), res_lens=i32(255, 3))
        if form == "lse":
            kw = dict(return_lse=True)
        if form == "tail":
            kw = dict(k_res=k_res[:, :100], v_res=v_res[:, :100])
        if form in ("ragged", "append", "rotary"):
            kw = dict(k_res=k_res, v_res=v_res, **lens)
        if form in ("append", "rotary"):
            kw.update(k_new=x["k"][:, :1], v_new=x["v"][:, :1])
        if form == "append":
            kw.update(advance=True)
        if form == "rotary":
            a = torch.arange(1024, device="cuda")[:, None] * torch.linspace(1, 0.01, 32, device="cuda")
            kw.update(rotary_cos=a.cos().to(q.dtype), rotary_sin=a.sin().to(q.dtype), rotary_interleaved=False)
        if form == "out32":
            kw = dict(out_dtype=torch.float32)
        if form == "splits":
            kw = dict(num_splits=3)
        if form == "bound":
            kw = dict(seqlen_k=300)
        if form == "paged":
            bufs, table = tuple(t.reshape(4, t.shape[1] // 2, *t.shape[2:]) for t in bufs[:3]) + (
                bufs[3].unflatten(3, (2, 256)).permute(0, 3, 1, 2, 4).reshape(4, *bufs[3].shape[1:3], 256),), i32(0, 1, 3, 2).view(2, 2)
        if form == "strided_q":
            q = torch.cat([q, q], 2)[:, :, 4:12]
        if form == "int_scale":
            scale = 1
        r = B.fwd_kvcache_int(q, *bufs, table, scale, "k-channel", group, bits, **kw)
        return [*(r if isinstance(r, tuple) else (r,)), *(t.view(torch.uint8) for t in bufs), k_res, v_res, *lens.values()]

    taken = []
    calls = I._calls()

    class Watched(I._InterpretedCalls):
        decode = staticmethod(lambda *a: taken.append(calls.decode(*a)) or taken[-1])
        pack = staticmethod(lambda *a: taken.append(calls.pack(*a)) or taken[-1])

    monkeypatch.setattr(I, "_CALLS", I._InterpretedCalls)
    python = outputs()                               # (also leaves a workspace for this layout)
    monkeypatch.setattr(I, "_CALLS", Watched)
    direct = outputs()
    assert len(taken) == 2 and all(t is not None for t in taken)
    assert len(python) == len(direct)
    for a, b in zip(python, direct):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


@pytest.mark.gpu
def test_refused_calls_are_still_refused():
    import bitladder_b200 as B
    x = H.gen_qkv(2, 256, 8, 2, seed=5)
    bufs = B.alloc_packed_cache(2, 256, 2, 128, 4, 128)
    q, k = x["q"].cuda(), x["k"].cuda()
    ok = lambda q=q, b=bufs, s=SCALE, g=128, **kw: B.fwd_kvcache_int(q, *b, None, s, "k-channel", g, 4, **kw)
    for call in (lambda: ok(q.float()), lambda: ok(q[:1]), lambda: ok(g=64), lambda: ok(q[..., ::2]), lambda: ok(seqlen_k=257),
                 lambda: ok(b=(bufs[0][:, :32], *bufs[1:])), lambda: ok(k_res=k), lambda: ok(k_res=k, v_res=k[:, ::2]),
                 lambda: ok(cache_seqlens=torch.zeros(2, dtype=torch.int64, device="cuda")), lambda: ok(out_dtype=torch.float64),
                 lambda: ok(k_new=k[:, :1], v_new=k[:, :1]), lambda: ok(cache_seqlens=torch.zeros(2, dtype=torch.int32)),
                 lambda: B.kvcache_pack_int(k[:, :100], bufs[0], bufs[1], k[:, :100], bufs[2], bufs[3], None, None, 100),
                 lambda: B.kvcache_pack_int(k, bufs[0], bufs[1], k.float(), bufs[2], bufs[3], None, None, 256),
                 lambda: B.kvcache_pack_int(k, bufs[0], bufs[1], k, bufs[2], bufs[3], None, None, 256, dst_token_offset=128)):
        with pytest.raises(RuntimeError):
            call()


@pytest.mark.gpu
def test_other_threads_run_during_a_launch(tmp_path):
    """A launch that waits (here: an entry point that sleeps) holds up its own thread only."""
    from bitladder_b200 import _lib, _torch_calls as T
    import bitladder_b200 as B
    source = tmp_path / "slow.c"
    source.write_text("#include <stddef.h>\n#include <unistd.h>\n"
                      "int slow(const void *a, void *s) { usleep(300000); return 0; }\nsize_t bytes(const void *a) { return 64; }\n")
    subprocess.run(["cc", "-shared", "-fPIC", "-o", str(tmp_path / "slow.so"), str(source)], check=True)
    slow, real = C.CDLL(str(tmp_path / "slow.so")), _lib.load()
    bind = lambda *f: T.bind(*(C.cast(x, C.c_void_p).value for x in f))
    x = {k: v.cuda() for k, v in H.gen_qkv(2, 256, 8, 2, seed=5).items() if isinstance(v, torch.Tensor)}
    bufs = B.alloc_packed_cache(2, 256, 2, 128, 4, 128)
    stream = torch.cuda.current_stream().cuda_stream
    spaces = {(0, stream): [torch.zeros(64, dtype=torch.uint8, device="cuda"), (2, 2, False)]}
    ticks, stop = [0], threading.Event()

    def tick():
        while not stop.is_set():
            time.sleep(0.002)
            ticks[0] += 1

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        bind(slow.slow, slow.slow, slow.bytes)
        for call in (lambda: T.step(0, 0), lambda: T.pack(x["k"], bufs[0], bufs[1], x["v"], bufs[2], bufs[3], "k-channel", 128, 4, 0, False),
                     lambda: T.decode(spaces, x["q"], *bufs, None, SCALE, "k-channel", 128, 4, None, None, None, None, None, True,
                                      None, 0, None, None, False, None, None, True)):
            before = ticks[0]
            assert call() is not None
            assert ticks[0] - before >= 20
    finally:
        bind(real.bd_decode, real.bd_pack, real.bd_decode_workspace_bytes)
        stop.set()
        thread.join()


def _small(B, seed=5):
    x = {k: v.cuda() for k, v in H.gen_qkv(2, 256, 8, 2, seed=seed).items() if isinstance(v, torch.Tensor)}
    bufs = B.alloc_packed_cache(2, 256, 2, 128, 4, 128)
    B.kvcache_pack_int(x["k"], bufs[0], bufs[1], x["v"], bufs[2], bufs[3], None, None, 256, "k-channel", 128, 4)
    torch.cuda.synchronize()
    return x, bufs


@pytest.mark.gpu
def test_side_streams_threads_and_captures(monkeypatch):
    """Calls on streams of their own, from threads of their own and into a graph give the bits of the Python path, each
    stream with its own workspace."""
    import bitladder_b200 as B
    from bitladder_b200 import bit_decode_interface as I
    sets = [_small(B, seed) for seed in (5, 6, 7)]
    decode = lambda x, bufs: B.fwd_kvcache_int(x["q"], *bufs, None, SCALE, "k-channel", 128, 4, num_splits=2, return_lse=True)
    calls = I._calls()
    monkeypatch.setattr(I, "_CALLS", I._InterpretedCalls)
    want = [[t.clone() for t in decode(*s)] for s in sets]
    torch.cuda.synchronize()
    monkeypatch.setattr(I, "_CALLS", calls)
    got = [None] * len(sets)

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(50):
                got[i] = decode(*sets[i])
            assert (0, stream.cuda_stream) in I._WORKSPACES
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, w in zip(got, want):
        assert all(torch.equal(a, b) for a, b in zip(g, w))
    stream, graph, (x, bufs) = torch.cuda.Stream(), torch.cuda.CUDAGraph(), sets[0]
    with torch.cuda.stream(stream):
        decode(x, bufs)                              # the stream's workspace is there before the capture
        stream.synchronize()
        taken = []
        monkeypatch.setattr(I, "_CALLS", type("Watched", (I._InterpretedCalls,), {
            "decode": staticmethod(lambda *a: taken.append(calls.decode(*a)) or taken[-1])}))
        with torch.cuda.graph(graph, stream=stream):
            out, lse = decode(x, bufs)
        assert taken[0] is not None
        q = x["q"].clone()
        for other, w in ((sets[1][0]["q"], None), (q, want[0])):
            x["q"].copy_(other)
            graph.replay()
            stream.synchronize()
            assert w is None or (torch.equal(out, w[0]) and torch.equal(lse, w[1]))


@pytest.mark.gpu
def test_misaligned_and_empty_tensors():
    """What the library refuses comes back to the Python path and is an error there; nothing to pack is none."""
    import bitladder_b200 as B
    x, bufs = _small(B)
    before = [t.clone() for t in bufs]
    shifted = lambda t: torch.cat([t.flatten(), t.flatten()[:8]])[1:1 + t.numel()].view(t.shape)
    pack = lambda k, v: B.kvcache_pack_int(k, bufs[0], bufs[1], v, bufs[2], bufs[3], None, None, k.shape[1], "k-channel", 128, 4)
    decode = lambda q, **kw: B.fwd_kvcache_int(q, *bufs, None, SCALE, "k-channel", 128, 4, **kw)
    for call in (lambda: pack(shifted(x["k"]), x["v"]), lambda: pack(x["k"], shifted(x["v"])), lambda: decode(shifted(x["q"])),
                 lambda: decode(x["q"], k_res=shifted(x["k"][:, :16].contiguous()), v_res=x["v"][:, :16].contiguous()),
                 lambda: decode(x["q"][:0]), lambda: pack(x["k"][:0], x["v"][:0])):
        with pytest.raises(RuntimeError):
            call()
    pack(x["k"][:, :0], x["v"][:, :0])
    assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(before, bufs))
    assert decode(x["q"], seqlen_k=0).abs().max() == 0

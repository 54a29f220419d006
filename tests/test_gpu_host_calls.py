"""The direct call path (arguments the kernels take as they are) and the converting one (constants
on the CPU, other layouts) give the same bits, and wrong arguments still raise."""

import threading
import time

import pytest
import torch

import flashquant_b200 as fq
from flashquant_b200 import kernels as K
from flashquant_b200 import workloads as W

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_direct_and_converting_calls_agree(consts, dtype):
    w = W.decode_workload(seq_lens=[1, 40, 700], num_q_heads=32, num_kv_heads=8, cfg=61, dtype=dtype)
    k, v = (t.to(DEV) for t in W.make_kv(w.total_tokens, 8, 128, 61, dtype))
    slots, bt, sl, q = (t.to(DEV) for t in (w.slot_mapping, w.block_table, w.seq_lens, w.q))
    host = [consts[n].contiguous() for n in ("rotation_128_0", "boundaries_128_3",
                                             "centroids_128_3", "boundaries_128_4",
                                             "centroids_128_4", "qjl_128_0")]
    got = []
    for c in (host, [t.to(DEV) for t in host]):
        rot, bk, ck, bv, cv, qjl = c
        cache = torch.zeros(w.num_blocks, 16, 8 * 136, dtype=torch.uint8, device=DEV)
        plane = torch.zeros(w.num_blocks, 16, 8 * 20, dtype=torch.uint8, device=DEV)
        fq.tq4_compress_append(k, v, cache, slots, rot, bk, bv)
        one = cache.clone()
        fq.tq4_compress_append_qjl(k, v, cache, plane, slots.int(), rot, bk, ck, bv, qjl)
        geo = (8, 128, 16)
        out = fq.split_k_paged_decode(q, cache, bt, sl, ck, cv, rot, *geo)
        multi = fq.split_k_paged_decode_multi(q[:, None].contiguous(), cache, bt, sl, ck, cv, rot,
                                              *geo)
        cu = torch.tensor([0, 1, 2, 3], dtype=torch.int32, device=DEV)
        pre = fq.paged_tq4_prefill(q, cache, bt, sl, cu, 1, ck, cv, rot, *geo)
        got.append((one, cache, plane, out, multi, pre))
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_strided_tokens_and_streams(consts):
    """Keys and values as slices of one projection, and a second stream with its own workspace."""
    rot, bk, bv = (consts[n].contiguous().to(DEV) for n in
                   ("rotation_128_0", "boundaries_128_3", "boundaries_128_4"))
    qkv = torch.randn(33, 3 * 8, 128, device=DEV).to(torch.bfloat16)
    k, v = qkv[:, 8:16], qkv[:, 16:]
    slots = torch.arange(33, device=DEV)
    a, b = (torch.zeros(3, 16, 8 * 136, dtype=torch.uint8, device=DEV) for _ in range(2))
    fq.tq4_compress_append(k, v, a, slots, rot, bk, bv)
    fq.tq4_compress_append(k.contiguous(), v.contiguous(), b, slots, rot, bk, bv)
    assert torch.equal(a, b)
    first = K.decode_workspace(torch.device(DEV), 1, 8, 8, 128, 0)
    with torch.cuda.stream(torch.cuda.Stream()):
        assert K.decode_workspace(torch.device(DEV), 1, 8, 8, 128, 0).data_ptr() != first.data_ptr()
    assert K.decode_workspace(torch.device(DEV), 1, 8, 8, 128, 0).data_ptr() == first.data_ptr()
    with pytest.raises(ValueError):
        fq.tq4_compress_append(k, v, a[..., :-1].contiguous(), slots, rot, bk, bv)


@pytest.mark.parametrize("n", [1, 40])
@pytest.mark.parametrize("b", [1, 3])
def test_attention_over_one_kv_head(consts, b, n):
    """One KV head: rows as the compressor returns them, turned so that the head dimension has a
    stride of its own, and part-filled buffers; constants on the device and on the CPU."""
    host = [consts[x].contiguous() for x in ("boundaries_128_4", "centroids_128_4", "rotation_128_0")]
    bnd, c, rot = (t.to(DEV) for t in host)
    q = torch.randn(b, 4, 1, 128, device=DEV).to(torch.float16)
    kv = []
    for _ in range(2):
        x = torch.randn(b * n, 1, 128, device=DEV).to(torch.float16)
        kv += [t.view(b, n, 1, -1).transpose(1, 2) for t in fq.tq4_compress(x, rot, bnd)]
    want = fq.fused_tq_attention(q, *(t.contiguous() for t in kv), c, c, rot)
    views = []
    for t in kv:
        buf = torch.zeros(b, 1, n + 7, t.shape[3], dtype=t.dtype, device=DEV)
        buf[:, :, :n] = t
        views.append(buf[:, :, :n])
    for cc, rr in ((c, rot), (host[1], host[2])):
        assert torch.equal(fq.fused_tq_attention(q, *kv, cc, cc, rr), want)
        assert torch.equal(fq.fused_tq_attention(q, *views, cc, cc, rr), want)
        assert torch.equal(fq.fused_tq_attention_kv(q, *views, cc, cc, rr, rr), want)
        assert torch.equal(fq.fused_tq_attention_kv(q, *kv, cc, cc, rr, rr), want)


def test_recorded_multi_token_call_after_a_larger_one(consts):
    """A call recorded in a CUDA graph on a stream that had run one before, then a call with a much wider
    block table on that stream: the replay writes nothing into memory that has been handed on."""
    w = W.decode_workload(seq_lens=[40, 700], num_q_heads=32, num_kv_heads=8, cfg=62)
    k, v = (t.to(DEV) for t in W.make_kv(w.total_tokens, 8, 128, 62))
    rot, bk, bv, ck, cv = (consts[n].contiguous().to(DEV) for n in (
        "rotation_128_0", "boundaries_128_3", "boundaries_128_4", "centroids_128_3", "centroids_128_4"))
    cache = torch.zeros(w.num_blocks, 16, 8 * 136, dtype=torch.uint8, device=DEV)
    fq.tq4_compress_append(k, v, cache, w.slot_mapping.to(DEV), rot, bk, bv)
    q = w.q.to(DEV)[:, None].repeat(1, 3, 1, 1)  # (three tokens: rows in scratch memory)
    table, lens = w.block_table.to(DEV), w.seq_lens.to(DEV)
    wide = torch.zeros(2, 100000, dtype=torch.int32, device=DEV)
    wide[:, :table.shape[1]] = table
    call = lambda t: fq.split_k_paged_decode_multi(q, cache, t, lens, ck, cv, rot, 8, 128, 16)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        want = call(table)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = call(table)
        assert torch.equal(call(wide), want)
        others = [torch.zeros(1 << 20, dtype=torch.uint8, device=DEV) for _ in range(8)]
        graph.replay()
        stream.synchronize()
        assert torch.equal(out, want)
        assert not any(bool(t.any()) for t in others)
    graph.reset()


def test_workspaces_stay_where_they_are():
    """The address that a recorded call holds: neither many streams nor a larger call moves it to
    other hands."""
    dev = torch.device(DEV)
    first = K.decode_workspace(dev, 1, 8, 8, 128, 0)
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(33)]
    with torch.cuda.stream(streams[0]):
        small = K.decode_workspace(dev, 1, 8, 8, 128, 0)
    at, size = small.data_ptr(), small.numel()
    del small
    for s in streams:
        with torch.cuda.stream(s):
            for use in (K._DECODE, K._ATTENTION):
                K._workspace(dev, use, 0)
    assert K.decode_workspace(dev, 1, 8, 8, 128, 0).data_ptr() == first.data_ptr()
    with torch.cuda.stream(streams[0]):
        assert K.decode_workspace(dev, 1, 8, 8, 128, 0).data_ptr() == at
        large = K._workspace(dev, K._DECODE, size + 1)
        assert large.data_ptr() != at and large.numel() >= 2 * size
        others = [torch.empty(1 << 20, dtype=torch.uint8, device=dev) for _ in range(16)]
    assert not any(t.data_ptr() < at + size and at < t.data_ptr() + t.numel() for t in others)


def test_attention_status_covers_all_streams():
    dev = torch.device(DEV)
    K._workspace(dev, K._ATTENTION, 0)
    with torch.cuda.stream(torch.cuda.Stream()):
        other = K._workspace(dev, K._ATTENTION, 0)
    assert K.attention_workspace_status(dev) == 0
    other[0] = 4
    assert K.attention_workspace_status(dev) == 4 and K.attention_workspace_status("cuda") == 4
    other[0] = 0
    assert K.attention_workspace_status(dev) == 0


def test_calls_without_the_extension_module(consts, monkeypatch):
    w = W.decode_workload(seq_lens=[40, 700], num_q_heads=32, num_kv_heads=8, cfg=63)
    k, v = (t.to(DEV) for t in W.make_kv(w.total_tokens, 8, 128, 63))
    rot, bk, bv, ck, cv = (consts[n].contiguous().to(DEV) for n in (
        "rotation_128_0", "boundaries_128_3", "boundaries_128_4", "centroids_128_3", "centroids_128_4"))

    def run():
        cache = torch.zeros(w.num_blocks, 16, 8 * 136, dtype=torch.uint8, device=DEV)
        fq.tq4_compress_append(k, v, cache, w.slot_mapping.to(DEV), rot, bk, bv)
        return cache, fq.split_k_paged_decode(w.q.to(DEV), cache, w.block_table.to(DEV),
                                              w.seq_lens.to(DEV), ck, cv, rot, 8, 128, 16)

    want = run()
    monkeypatch.setattr(K, "_host_module", K._ConvertingCalls())
    assert all(torch.equal(a, b) for a, b in zip(run(), want))
    ws = K.decode_workspace(torch.device(DEV), 2, 32, 8, 128, 0)
    assert ws.data_ptr() == K.decode_workspace(torch.device(DEV), 2, 32, 8, 128, 0).data_ptr()
    assert K.attention_workspace_status(DEV) == 0


def test_other_threads_run_while_a_call_waits(consts):
    """A launch queue that is full behind half a second of other work makes a call wait; the
    interpreter lock is free meanwhile."""
    rot, bk = (consts[n].contiguous().to(DEV) for n in ("rotation_128_0", "boundaries_128_3"))
    k = torch.randn(4, 8, 128, device=DEV).to(torch.bfloat16)
    cache = torch.zeros(1, 16, 8 * 136, dtype=torch.uint8, device=DEV)
    slots = torch.arange(4, device=DEV)
    fq.tq4_compress_append(k, k, cache, slots, rot, bk)
    torch.cuda.synchronize()
    seen, stop = [], threading.Event()

    def watch():
        while not stop.is_set():
            seen.append(time.perf_counter())
            time.sleep(0.001)

    watcher = threading.Thread(target=watch)
    watcher.start()
    try:
        torch.cuda._sleep(10 ** 9)  # about 0.5 s on the stream
        longest = 0.0
        for _ in range(4000):
            t = time.perf_counter()
            fq.tq4_compress_append(k, k, cache, slots, rot, bk)
            longest = max(longest, time.perf_counter() - t)
        torch.cuda.synchronize()
    finally:
        stop.set()
        watcher.join()
    assert longest > 0.2, f"no call waited ({longest:.3f} s): the queue was not full"
    gap = max(b - a for a, b in zip(seen, seen[1:]))
    assert gap < 0.1, f"no other thread ran for {gap:.3f} s"


def test_threads_on_one_stream(consts):
    """Single-token attention of two threads on one stream, which share a workspace: a call is several
    launches, and nothing of another call comes in between."""
    bnd, c, rot = (consts[n].contiguous().to(DEV) for n in ("boundaries_128_4", "centroids_128_4", "rotation_128_0"))
    cases = []
    for i in range(2):
        x = torch.randn(2 * 8 * 600, 1, 128, device=DEV, generator=torch.Generator(DEV).manual_seed(i)).half()
        p, n = fq.tq4_compress(x, rot, bnd)
        q = torch.randn(2, 32, 1, 128, device=DEV).half()
        args = (q, p.view(2, 8, 600, 64), n.view(2, 8, 600, 1), p.view(2, 8, 600, 64), n.view(2, 8, 600, 1), c, c, rot)
        cases.append((args, fq.fused_tq_attention(*args)))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    wrong = []

    def run(args, want):
        with torch.cuda.stream(stream):
            outs = [fq.fused_tq_attention(*args) for _ in range(300)]
            wrong.extend(i for i, o in enumerate(outs) if not torch.equal(o, want))

    threads = [threading.Thread(target=run, args=case) for case in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_every_call_both_ways(consts, monkeypatch):
    """The entry points that the extension module takes, and the same through ctypes: the same bits."""
    w = W.decode_workload(seq_lens=[1, 40, 700], num_q_heads=32, num_kv_heads=8, cfg=64)
    k, v = (t.to(DEV) for t in W.make_kv(w.total_tokens, 8, 128, 64))
    rot, bk, bv, ck, cv, qjl = (consts[n].contiguous().to(DEV) for n in (
        "rotation_128_0", "boundaries_128_3", "boundaries_128_4", "centroids_128_3", "centroids_128_4",
        "qjl_128_0"))
    rt = rot.T.contiguous()
    even, odd = rt[:, 0::2].contiguous(), rt[:, 1::2].contiguous()
    slots, bt, sl, q = (t.to(DEV) for t in (w.slot_mapping, w.block_table, w.seq_lens, w.q))
    geo = (8, 128, 16)
    x = torch.randn(2, 8, 50, 128, device=DEV).to(torch.bfloat16)
    one = torch.randn(2, 32, 1, 128, device=DEV).to(torch.bfloat16)
    many = torch.randn(2, 32, 50, 128, device=DEV).to(torch.bfloat16)

    def run():
        out = list(fq.tq4_compress(k, rot, bk, rotation_T_even=even, rotation_T_odd=odd))
        cache = torch.zeros(w.num_blocks, 16, 8 * 136, dtype=torch.uint8, device=DEV)
        plane = torch.zeros(w.num_blocks, 16, 8 * 20, dtype=torch.uint8, device=DEV)
        fq.tq4_compress_append_qjl(k, v, cache, plane, slots, rot, bk, ck, bv, qjl)
        out += [cache, plane, fq.split_k_paged_decode_qjl(q, cache, plane, bt, sl, ck, cv, rot, qjl, *geo)]
        tables = (even, odd, bv, cv, rot)
        for new in (1, 50):
            bufs = [torch.zeros(2, 8, 64, n, dtype=t, device=DEV) for n, t in
                    ((64, torch.uint8), (1, torch.float32)) * 2]
            K.cache_update(x[:, :, :new].contiguous(), x[:, :, -new:].contiguous(), tables, tables, *bufs, 3)
            views = [t[:, :, :3 + new] for t in bufs]
            out += bufs + [fq.fused_tq_attention_kv(one, *views, cv, cv, rot, rot)]
            read = [torch.zeros(2, 8, 64, 128, dtype=x.dtype, device=DEV) for _ in range(2)]
            ws = torch.empty(2 * 8 * new * 128 * 4, dtype=torch.uint8, device=DEV)
            K.cache_update(x[:, :, :new].contiguous(), x[:, :, -new:].contiguous(), tables, tables, *bufs, 3,
                           *read, 5, ws)
            out += bufs + read
        return out + [fq.fused_tq_attention(many, *(t[:, :, 3:53] for t in bufs), cv, cv, rot, is_causal=True)]

    direct = run()
    monkeypatch.setattr(K, "_host_module", K._ConvertingCalls())
    for i, (a, b) in enumerate(zip(direct, run())):
        assert torch.equal(a, b), i

"""Kernels that start before their predecessor in the stream has finished: chains in which every kernel reads what the one
before it wrote and overwrites what the one before that read, enqueued without a pause, against the same calls one at a time."""
import ctypes

import pytest
import torch

from cai_b200 import ops

pytestmark = pytest.mark.gpu


def _chain(x, w_gu, w_down, gain, y, dw):
    """Norm, gate/up product, SwiGLU, down product with the residual added, weight gradient, and back to the norm's gradient."""
    n, rstd = ops.rmsnorm_fwd(x, gain)
    gu = ops.gemm(n, w_gu)
    act = ops.swiglu_fwd(gu)
    ops.gemm(act, w_down, out=y, residual=x)
    ops.gemm(y, act, trans_a=True, trans_b=True, out=dw, accumulate=True)
    dact = ops.gemm(y, w_down, trans_b=True)
    dgu = ops.swiglu_bwd(gu, dact)
    dn = ops.gemm(dgu, w_gu, trans_b=True)
    dx, dg = ops.rmsnorm_bwd(x, gain, rstd, dn)
    x.copy_(dx)          # a kernel of another library between two of ours, and the buffer the first one read is overwritten
    return dg


def _inputs(rows, hidden, ffn):
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).bfloat16()
    return (r(rows, hidden), r(2 * ffn, hidden, std=0.05), r(hidden, ffn, std=0.05), 1 + r(hidden, std=0.1), r(rows, hidden),
            torch.zeros(hidden, ffn, device="cuda"))


# one tile and split products, several waves of pairs, rows that leave a last tile almost empty
@pytest.mark.parametrize("rows,hidden,ffn", [(8, 128, 128), (264, 256, 512), (1000, 1000, 1368), (5000, 1024, 3072)])
@pytest.mark.parametrize("captured", [False, True])
def test_chain_matches_one_call_at_a_time(rows, hidden, ffn, captured, monkeypatch):
    args = _inputs(rows, hidden, ffn)
    start = [a.clone() for a in args]

    def reset():
        for a, s in zip(args, start):
            a.copy_(s)

    real = {n: getattr(ops, n) for n in ("rmsnorm_fwd", "gemm", "swiglu_fwd", "swiglu_bwd", "rmsnorm_bwd")}

    def waiting(f):
        def call(*a, **k):
            out = f(*a, **k)
            torch.cuda.synchronize()
            return out
        return call

    for n, f in real.items():
        monkeypatch.setattr(ops, n, waiting(f))
    gains = [_chain(*args).clone() for _ in range(3)]
    want = [a.clone() for a in args] + gains
    for n, f in real.items():
        monkeypatch.setattr(ops, n, f)

    for _ in range(5):
        reset()
        if captured:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                got_gains = [_chain(*args) for _ in range(3)]
            graph.replay()
        else:
            got_gains = [_chain(*args) for _ in range(3)]
        torch.cuda.synchronize()
        for got, ref in zip(list(args) + got_gains, want):
            assert torch.equal(got, ref)


@pytest.mark.parametrize("batch,seq,heads,kv_heads", [(1, 128, 2, 1), (2, 384, 6, 2), (8, 384, 12, 4), (1, 2048, 8, 8)])
def test_attention_chain_matches_one_call_at_a_time(batch, seq, heads, kv_heads):
    g = torch.Generator(device="cuda").manual_seed(seq)
    qkv0 = torch.randn(batch * seq, (heads + 2 * kv_heads) * 128, generator=g, device="cuda").bfloat16()
    dout = torch.randn(batch * seq, heads * 128, generator=g, device="cuda").bfloat16()
    table = ops.rope_table(seq, 128)

    def steps(sync):
        qkv = qkv0.clone()
        outs = []
        for _ in range(3):
            ops.rope_apply_(qkv, table, seq, heads, kv_heads, 128)
            sync()
            out, lse = ops.flash_attn_fwd(qkv, batch, seq, heads, kv_heads, 128)
            sync()
            dqkv = ops.flash_attn_bwd(qkv, out, dout, lse, batch, seq, heads, kv_heads, 128)
            sync()
            ops.rope_apply_(dqkv, table, seq, heads, kv_heads, 128, inverse=True)
            sync()
            qkv = dqkv                       # the next round rotates and reads what this one wrote
            outs += [out, lse]
        torch.cuda.synchronize()
        return outs + [qkv]

    want = steps(torch.cuda.synchronize)
    for _ in range(5):
        for got, ref in zip(steps(lambda: None), want):
            assert torch.equal(got, ref)


def _early_launches(call):
    """How many launches of `call`, captured, may start before their predecessor has ended (programmatic edges of the graph)."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    get = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2     # (graph, from, to, {from_port, to_port, type, ...}, count)
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert get(handle, None, None, None, ctypes.byref(n)) == 0
    nodes, data = (ctypes.c_void_p * n.value)(), ((ctypes.c_ubyte * 8) * n.value)()
    assert get(handle, nodes, (ctypes.c_void_p * n.value)(), data, ctypes.byref(n)) == 0
    return sum(d[2] == 1 for d in data)


# Under a limit no launch starts early: turns of the split form, and products behind each other in the persistent one.
@pytest.mark.parametrize("M,N,K", [(333, 1024, 3000), (300, 968, 2048), (1536, 1536, 520), (4096, 4104, 264)])
def test_limited_products_start_behind_each_other(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)

    def twice(limit):
        ops.gemm(a, b, out=out, sm_limit=limit)
        ops.gemm(a, b, out=out, sm_limit=limit)

    assert _early_launches(lambda: twice(0)) > 0
    for limit in (2, 10, 60):
        assert _early_launches(lambda: twice(limit)) == 0


# The SMs that a product does not fill, under a limit or for want of tiles, stay free until it ends: a product of another stream, whose
# CTAs share an SM with no other product's, is done long before, although the next one of the first stream is already enqueued.
@pytest.mark.parametrize("M,N,K,limit", [(4096, 4096, 4096, 32), (256, 256, 262144, 0)])
def test_sms_beside_a_product_stay_free(M, N, K, limit):
    g = torch.Generator(device="cuda").manual_seed(0)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    wide = torch.randn(4096, 4096, generator=g, device="cuda").bfloat16()
    small = wide[:1024, :1024]
    out, out_wide, out_small = (torch.empty(n, m, device="cuda", dtype=torch.bfloat16) for n, m in ((M, N), (4096, 4096), (1024, 1024)))
    main, beside = torch.cuda.Stream(), torch.cuda.Stream()
    start, alone, done = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    torch.cuda.synchronize()

    def run(both):
        with torch.cuda.stream(main):
            torch.cuda._sleep(400000)          # all of it is enqueued meanwhile
            start.record()
            ops.gemm(a, b, out=out, sm_limit=limit)
            if both:
                ops.gemm(wide, wide, out=out_wide)
            else:
                alone.record()
        if both:
            with torch.cuda.stream(beside):
                beside.wait_event(start)
                torch.cuda._sleep(60000)       # the first product has started
                ops.gemm(small, small, out=out_small)
                done.record()
        torch.cuda.synchronize()
        return start.elapsed_time(done if both else alone)

    first, beside_it = (sorted(run(both) for _ in range(7))[3] for both in (False, True))
    assert beside_it < 0.6 * first

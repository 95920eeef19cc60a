"""Kernels that start before their predecessor in the stream has finished: chains in which every kernel reads what the one
before it wrote and overwrites what the one before that read, enqueued without a pause, against the same calls one at a time."""
import ctypes
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from cai_b200 import ops
from cai_b200.ops._lib import check, lib

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


def _agrees_with_one_call_at_a_time(steps, rounds=5):
    """`steps(sync)` runs a chain from its own start state, calling `sync` behind every op, and returns what it wrote."""
    want = steps(torch.cuda.synchronize)
    for _ in range(rounds):
        got = steps(lambda: None)
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


# Weights added up, quantised by blocks and multiplied with rows quantised just before, the result quantised and multiplied back into the
# buffer that the first op read. The product on one CTA a tile and on pairs; weights on 16 bytes and not.
@pytest.mark.parametrize("M,N,K,offset", [(128, 28672, 1152, 0), (300, 640, 1024, 0), (300, 640, 1024, 1)])
def test_e4m3_chain_matches_one_call_at_a_time(M, N, K, offset):
    g = torch.Generator(device="cuda").manual_seed(M)
    x0 = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w0 = (torch.randn(N, K, generator=g, device="cuda") * 0.02).bfloat16()
    wide = torch.empty(N, K + 8, device="cuda", dtype=torch.bfloat16)

    def steps(sync):
        x, w, outs = x0.clone(), w0.clone(), []
        for _ in range(3):
            check(lib().cai_add_bf16(w.data_ptr(), w0.data_ptr(), w.data_ptr(), w.numel(), torch.cuda.current_stream().cuda_stream), "add")
            sync()
            wide[:, offset:offset + K].copy_(w)
            wq, ws, wtq, wts = ops.quant_blocks_128x128(wide[:, offset:offset + K], transposed=True)
            sync()
            xq, xs = ops.quant_rows_1x128(x)
            sync()
            y = ops.gemm_fp8(xq, xs, wq, ws)
            sync()
            yq, ys = ops.quant_rows_1x128(y)
            sync()
            ops.gemm_fp8(yq, ys, wtq, wts, out=x)
            sync()
            outs += [y, wq, wtq]
        return outs + [x, w]

    _agrees_with_one_call_at_a_time(steps)


# The expert half of a layer on the counts that the router has just written, its logits changed by their gradient: every expert's rows in a
# slab of their own, and eight slabs to a group.
@pytest.mark.parametrize("groups", [32, 4])
def test_expert_chain_matches_one_call_at_a_time(groups):
    T, E, k, H, F, cap = 512, 32, 2, 256, 512, 128
    M = E // groups * cap
    g = torch.Generator(device="cuda").manual_seed(groups)
    r = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).bfloat16()
    logits0, dw = torch.randn(T, E, generator=g, device="cuda"), torch.randn(T, k, generator=g, device="cuda")
    x, dy, wgu, wd = r(E * cap, H), r(E * cap, H), r(groups * 2 * F, H, std=0.05), r(groups * H, F, std=0.05)
    z = lambda rows, cols, dtype=torch.bfloat16: torch.zeros(rows, cols, device="cuda", dtype=dtype)

    def steps(sync):
        logits, outs = logits0.clone(), []
        gu, y, dact, dx = z(E * cap, 2 * F), z(E * cap, H), z(E * cap, F), z(E * cap, H)
        dwd, dwgu = z(groups * H, F, torch.float32), z(groups * 2 * F, H, torch.float32)
        for _ in range(3):
            idx, w, pos, counts = ops.moe_route_fwd(logits, k, cap)
            sync()
            rows = dict(groups=groups, seg_counts=counts, seg_rows=cap, seg_mode=1)
            depth = dict(groups=groups, seg_counts=counts, seg_rows=cap, seg_mode=2, trans_a=True, trans_b=True, accumulate=True)
            ops.gemm_grouped(x, wgu, gu, M, 2 * F, H, **rows)
            sync()
            act = ops.swiglu_fwd(gu)
            sync()
            ops.gemm_grouped(act, wd, y, M, H, F, **rows)
            sync()
            ops.gemm_grouped(y, wd, dact, M, F, H, trans_b=True, **rows)
            sync()
            ops.gemm_grouped(dy, act, dwd, H, F, M, **depth)
            sync()
            dgu = ops.swiglu_bwd(gu, dact)
            sync()
            ops.gemm_grouped(dgu, wgu, dx, M, H, 2 * F, trans_b=True, **rows)
            sync()
            ops.gemm_grouped(dgu, x, dwgu, 2 * F, H, M, **depth)
            sync()
            logits += ops.moe_route_bwd(logits, idx, dw, pos)
            sync()
            outs += [idx, w, pos, counts, act, dgu]
        return outs + [gu, y, dact, dx, dwd, dwgu, logits]

    _agrees_with_one_call_at_a_time(steps)


# Embedding, norm, logits, softmax cross-entropy (whole rows, and in the pieces of a vocabulary-parallel head), the gradients, AdamW, and again
# with the parameters it wrote. The loss is an atomic sum and is compared within its rounding.
@pytest.mark.parametrize("pieces", [False, True])
@pytest.mark.parametrize("T,V,H", [(256, 512, 256), (1920, 5000, 1000)])
def test_head_chain_matches_one_call_at_a_time(T, V, H, pieces):
    g = torch.Generator(device="cuda").manual_seed(V)
    tokens, targets = (torch.randint(0, V, (T,), generator=g, device="cuda", dtype=torch.int32) for _ in range(2))
    master0 = torch.randn(V, H, generator=g, device="cuda") * 0.05
    gain = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).bfloat16()
    L, losses = lib(), []
    P, I, LL, F32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    L.cai_ce_rowmax.argtypes = [P, P, I, I, LL, P]
    L.cai_ce_rowsum.argtypes = [P, P, P, I, I, LL, P]
    L.cai_ce_grad_tp.argtypes = [P, P, P, P, P, I, I, LL, I, I, F32, F32, P]

    def steps(sync):
        master, m, v, grad = master0.clone(), torch.zeros_like(master0), torch.zeros_like(master0), torch.empty_like(master0)
        param, loss, outs = master.bfloat16(), torch.zeros(1, device="cuda"), []
        st = torch.cuda.current_stream().cuda_stream
        for step in range(1, 4):
            h = ops.embed_fwd(tokens, param)
            sync()
            n, rstd = ops.rmsnorm_fwd(h, gain)
            sync()
            logits = ops.gemm(n, param)
            sync()
            if pieces:
                top, total = torch.empty(T, device="cuda"), torch.empty(T, device="cuda")
                check(L.cai_ce_rowmax(logits.data_ptr(), top.data_ptr(), T, V, V, st), "rowmax")
                sync()
                check(L.cai_ce_rowsum(logits.data_ptr(), top.data_ptr(), total.data_ptr(), T, V, V, st), "rowsum")
                sync()
                check(L.cai_ce_grad_tp(logits.data_ptr(), targets.data_ptr(), top.data_ptr(), total.data_ptr(), loss.data_ptr(), T, V, V, 0, 1,
                                       1.0 / T, 1.0 / T, st), "grad_tp")
            else:
                ops.cross_entropy_(logits, targets, loss, grad_scale=1.0 / T, loss_scale=1.0 / T)
            sync()
            ops.gemm(logits, n, trans_a=True, trans_b=True, out=grad)
            sync()
            dn = ops.gemm(logits, param, trans_b=True)
            sync()
            dh, dgain = ops.rmsnorm_bwd(h, gain, rstd, dn)
            sync()
            ops.embed_bwd_(tokens, dh, grad)
            sync()
            ops.adamw_(master, m, v, grad, param, step, lr=1e-2)
            sync()
            outs += [h, logits, dh, dgain]
        losses.append(loss)
        return outs + [master, m, v, grad, param]

    _agrees_with_one_call_at_a_time(steps)
    # three means of T losses of about log V, each added in fp32 in any order
    values = torch.cat(losses).double()
    assert (values.max() - values.min()).item() <= 3 * T * 2.0 ** -24 * values.max().item()


# A whole step, as the executor enqueues it, against the same with every launch waited for: the same parameters and gradients.
@pytest.mark.parametrize("config", ["tiny.cfg", "tiny_moe.cfg"])
def test_step_matches_one_launch_at_a_time(config):
    code = ("import hashlib, sys, torch\n"
            "from cai_b200.runtime.engine import Engine, synthetic_batch\n"
            "e = Engine(sys.argv[1], rank=0, world=1, local_rank=0)\n"
            "for i in range(4):\n"
            "    e.step(*synthetic_batch(e.model.vocab_size, e.model.seq_len, e.hdr.num_microbatches * e.model.microbatch, step=i, seed=3))\n"
            "h = hashlib.sha256()\n"
            "for n in ('grad', 'param', 'master', 'm', 'v'):\n"
            "    h.update(e.view('@flat_' + n).contiguous().view(torch.uint8).cpu().numpy().tobytes())\n"
            "print(h.hexdigest())\n"
            "e.close()\n")
    root = Path(__file__).resolve().parent.parent
    digests = []
    for blocking in ("0", "1"):
        r = subprocess.run([sys.executable, "-c", code, str(root / "configs" / config)], capture_output=True, text=True, cwd=root, timeout=300,
                           env=dict(os.environ, CUDA_LAUNCH_BLOCKING=blocking))
        assert r.returncode == 0, r.stderr[-2000:]
        digests.append(r.stdout.strip().splitlines()[-1])
    assert digests[0] == digests[1]


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

"""What the framework's speed is measured on: the work a training job gives it, through its public entry points.

Six kinds of case, each with its inputs, the call, the least traffic and arithmetic it needs, and a tolerance:

  step        one optimizer step of a decoder through ``Engine.step``: the batch is copied from pinned host memory, every
              microbatch runs forward and backward, AdamW updates the parameters, the loss is read back. Dense models in bf16 or
              with e4m3 linear layers, with and without activation recompute, tied or untied embeddings; a stream of batches.
  linear      a linear layer written on ``cai_b200.ops``: output (optionally with the residual added), input gradient, weight
              gradient in fp32 (first microbatch: written; later ones: accumulated).
  linear_fp8  the same layer in e4m3: the activations are quantised on the way in, the weights were quantised once.
  experts     the expert half of a mixture-of-experts layer: softmax top-k router, grouped gate / up and down projections over
              ragged slabs, SwiGLU, and the gradients of all of them. (A whole step of such a model sends near-tied tokens to other
              experts after any change of rounding, which no tolerance on its results describes; here the logits are given.)
  attention   rotary embedding, causal grouped-query attention forward and backward, inverse rotary embedding.
  head        the end of a decoder: final norm, vocabulary projection, softmax cross-entropy, and the gradients of all three.
"""
import math

import torch

from cai_b200 import ops
from cai_b200.runtime.engine import Engine, synthetic_batch

BATCHES = 4          # different batches a training state cycles through

STEP = dict(kind="step", param_dtype="bf16", recompute=0, tie_embeddings=0, lr=3e-4)


def listed():
    return [
        # the smallest training step: the model of configs/tiny.cfg, what a test, a smoke run or a hyper-parameter search on a
        # toy model executes thousands of times; bound by launches and the host path
        dict(STEP, name="step_tiny", hidden_size=256, ffn_hidden=512, num_layers=2, num_heads=2, num_kv_heads=1, vocab_size=512,
             seq_len=128, microbatch=2, grad_accum=2, lr=1e-3),
        # a small model with widths that divide nothing in particular, tied embeddings, recompute: research-sized training
        dict(STEP, name="step_small_ragged", hidden_size=1000, ffn_hidden=2728, num_layers=6, num_heads=9, num_kv_heads=3,
             vocab_size=5000, seq_len=640, microbatch=3, grad_accum=2, recompute=1, tie_embeddings=1),
        # the benchmark model's widths (configs/b200_tp8.cfg) with half of its layers, four microbatches of 4096 tokens
        dict(STEP, name="step_dense", hidden_size=2048, ffn_hidden=8192, num_layers=12, num_heads=16, num_kv_heads=8,
             vocab_size=32000, seq_len=4096, microbatch=1, grad_accum=4),
        # two layers of the 8B-class model with e4m3 linear layers (configs/b200_fsdp8b.cfg): wide layers, large vocabulary
        dict(STEP, name="step_fp8_8b_layers", param_dtype="fp8e4m3", hidden_size=4096, ffn_hidden=14336, num_layers=2, num_heads=32,
             num_kv_heads=8, vocab_size=128256, seq_len=8192, microbatch=1, grad_accum=1),
        # the expert layers of the two mixture-of-experts models (configs/tiny_moe.cfg, configs/b200_moe_ep8.cfg), all experts here
        dict(kind="experts", name="experts_tiny", tokens=512, experts=32, top_k=2, hidden=256, ffn=512),
        dict(kind="experts", name="experts_64", tokens=8192, experts=64, top_k=8, hidden=4096, ffn=1536),
        # a layer on few tokens (a short fine-tuning batch), odd row count
        dict(kind="linear", name="linear_few_rows", rows=333, in_features=1024, out_features=3000, residual=1, accumulate=0),
        # gate / up projection of the benchmark model on one launch of 16384 tokens, later microbatches
        dict(kind="linear", name="linear_large", rows=16384, in_features=2048, out_features=16384, residual=0, accumulate=1),
        # a down projection of the 8B-class model on a mid-sized batch, e4m3
        dict(kind="linear_fp8", name="linear_fp8_mid", rows=2000, in_features=14336, out_features=4096),
        # many short sequences, and one long one at the 8B-class model's heads
        dict(kind="attention", name="attention_short", batch=8, seq=384, heads=12, kv_heads=4),
        dict(kind="attention", name="attention_long", batch=1, seq=8192, heads=32, kv_heads=8),
        # the benchmark model's head on one 4096-token chunk
        dict(kind="head", name="head_32k", rows=4096, hidden=2048, vocab=32000),
    ]


# ---------------------------------------------------------------------------- more cases of the same ranges
MOST_FLOPS = 9.0e13      # the largest listed step
MOST_BYTES = 4.5e10
MOST_PARAMS = 9.0e8


def _log(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / multiple)) * multiple))


def _draw_step(rng, flavour):
    c = dict(STEP)
    c["num_kv_heads"] = rng.choice([1, 2, 4, 8])
    c["num_heads"] = c["num_kv_heads"] * rng.choice([1, 2, 3, 4])
    c["seq_len"] = _log(rng, 128, 4096, 128)
    c["microbatch"] = rng.choice([1, 2, 3, 4])
    c["grad_accum"] = rng.choice([1, 2, 3, 4, 8])
    c["vocab_size"] = _log(rng, 512, 32000, 8)
    if flavour == "fp8":
        c.update(param_dtype="fp8e4m3", hidden_size=_log(rng, 256, 4096, 128), ffn_hidden=_log(rng, 512, 14336, 128),
                 num_layers=rng.choice([1, 2, 3, 4]))
    else:
        # rounded widths as often as odd ones
        m = rng.choice([8, 128])
        c.update(hidden_size=_log(rng, 128, 3072, m), num_layers=_log(rng, 1, 12), recompute=int(rng.random() < 0.25),
                 tie_embeddings=int(rng.random() < 0.25))
        c["ffn_hidden"] = min(12288, max(256, int(c["hidden_size"] * rng.uniform(2.0, 4.0)) // m * m))
    return c


def draw(rng):
    while True:
        kind = rng.choices(["dense", "fp8", "linear", "linear_fp8", "experts", "attention", "head"], [7, 2, 3, 2, 3, 4, 2])[0]
        if kind in ("dense", "fp8"):
            c = _draw_step(rng, kind)
            if _step_params(c)[0] > MOST_PARAMS or _step_tokens(c) > 16384:
                continue
        elif kind in ("linear", "linear_fp8"):
            m = 128 if kind == "linear_fp8" else 8
            c = dict(kind=kind, rows=_log(rng, 16, 16384), in_features=_log(rng, 128, 16384, m), out_features=_log(rng, 128, 16384, m))
            if kind == "linear":
                c.update(residual=int(rng.random() < 0.5), accumulate=int(rng.random() < 0.5))
        elif kind == "experts":
            c = dict(kind=kind, tokens=_log(rng, 128, 8192), experts=rng.choice([32, 64, 128]), top_k=rng.choice([1, 2, 4, 6, 8]),
                     hidden=_log(rng, 256, 4096, 64), ffn=_log(rng, 128, 1536, 64))
            if c["experts"] * c["hidden"] * c["ffn"] > 64 * 4096 * 1536:
                continue
        elif kind == "attention":
            kv = rng.choice([1, 2, 4, 8])
            c = dict(kind=kind, batch=_log(rng, 1, 16), seq=_log(rng, 128, 8192, 128), heads=kv * rng.choice([1, 2, 3, 4]), kv_heads=kv)
            if c["batch"] * c["seq"] > 32768:
                continue
        else:
            c = dict(kind=kind, rows=_log(rng, 64, 8192), hidden=_log(rng, 256, 4096, 8), vocab=_log(rng, 512, 128256, 8))
            if c["rows"] * c["vocab"] > 4096 * 128256:
                continue
        w = work(c)
        if w["flops"] <= MOST_FLOPS and w["bytes"] <= MOST_BYTES:
            return c


# ---------------------------------------------------------------------------- inputs
def _config_text(c, seed):
    keys = ("hidden_size", "ffn_hidden", "num_layers", "num_heads", "num_kv_heads", "vocab_size", "seq_len", "param_dtype",
            "recompute", "tie_embeddings", "microbatch", "grad_accum", "lr")
    text = "".join(f"{k} = {c[k]}\n" for k in keys)
    return text + (f"is_moe = 0\nhead_dim = 128\ntp = 1\npp = 1\nep = 1\noptim_dtype = fp32\nseed = {seed % 1000003}\n"
                   "gpus_per_rack = 1\ntrays_per_rack = 1\ngpus_per_tray = 1\nnum_racks = 1\n")


def prepare(case, seed):
    c = case
    if c["kind"] == "step":
        # An engine clears its arena on the caller's stream and fills it on its own. The clearing is waited for before the
        # parameters are drawn and the rotary table is laid down, so that a large arena is not cleared over them.
        eng = Engine(config_text=_config_text(c, seed), rank=0, world=1, local_rank=0, init_params=False)
        torch.cuda.synchronize()
        table = ops.rope_table(c["seq_len"], 128, theta=eng.train.rope_theta).view(-1)
        eng.view("@rope_table").view(-1)[:table.numel()].copy_(table)
        torch.cuda.synchronize()
        eng.init_parameters()
        rows = c["microbatch"] * c["grad_accum"]
        batches = [synthetic_batch(c["vocab_size"], c["seq_len"], rows, step=i, seed=seed % 1000003) for i in range(BATCHES)]
        state = {k: eng.view("@flat_" + k) for k in ("grad", "param", "master", "m", "v")}
        return dict(kind="step", engine=eng, batches=batches, at=0, state=state)

    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))

    def normal(*shape, std=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * std).to(torch.bfloat16)

    s = dict(c)
    if c["kind"] == "linear":
        M, K, N = c["rows"], c["in_features"], c["out_features"]
        s.update(x=normal(M, K), w=normal(N, K, std=0.02), dy=normal(M, N, std=0.01), dw=torch.zeros(N, K, device="cuda"),
                 res=normal(M, N) if c["residual"] else None)
    elif c["kind"] == "linear_fp8":
        M, K, N = c["rows"], c["in_features"], c["out_features"]
        s.update(x=normal(M, K), dy=normal(M, N, std=0.01), w=ops.quant_blocks_128x128(normal(N, K, std=0.02), transposed=True))
    elif c["kind"] == "experts":
        T, E, k, H, F = c["tokens"], c["experts"], c["top_k"], c["hidden"], c["ffn"]
        cap = (2 * T * k // E + 127) // 128 * 128      # room for twice the average load, as the plan compiler gives a slab
        s.update(cap=cap, logits=torch.randn(T, E, generator=g, device="cuda"), dw=torch.randn(T, k, generator=g, device="cuda") * 0.01)
        # tokens in their experts' slabs (rows past an expert's load are zero), as a dispatch leaves them
        idx, _, pos, counts = ops.moe_route_fwd(s["logits"], k, cap)
        kept = pos.view(-1) >= 0
        row = (idx.view(-1).long() * cap + pos.view(-1))[kept]
        tok = (torch.arange(T * k, device="cuda") // k)[kept]
        xs, dys = (torch.zeros(E * cap, H, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        xs[row] = normal(T, H)[tok]
        dys[row] = normal(T, H, std=0.01)[tok]
        s.update(live=counts.clamp(max=cap), xs=xs, dys=dys, wgu=normal(E * 2 * F, H, std=0.02), wd=normal(E * H, F, std=0.02))
        # results of the grouped products; rows of empty tiles stay as they are
        for name, rows, cols, dtype in (("gu", E * cap, 2 * F, torch.bfloat16), ("y", E * cap, H, torch.bfloat16),
                                        ("dact", E * cap, F, torch.bfloat16), ("dx", E * cap, H, torch.bfloat16),
                                        ("dwd", E * H, F, torch.float32), ("dwgu", E * 2 * F, H, torch.float32)):
            s[name] = torch.zeros(rows, cols, device="cuda", dtype=dtype)
    elif c["kind"] == "attention":
        T, nh, nkv = c["batch"] * c["seq"], c["heads"], c["kv_heads"]
        s.update(qkv=normal(T, (nh + 2 * nkv) * 128), dout=normal(T, nh * 128, std=0.1), table=ops.rope_table(c["seq"], 128))
    else:
        T, H, V = c["rows"], c["hidden"], c["vocab"]
        s.update(h=normal(T, H), gain=(1 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(torch.bfloat16),
                 w=normal(V, H, std=0.02), targets=torch.randint(0, V, (T,), generator=g, device="cuda", dtype=torch.int32))
    return s


# ---------------------------------------------------------------------------- the calls
def _run_step(s):
    tokens, targets = s["batches"][s["at"] % BATCHES]
    s["at"] += 1
    loss = s["engine"].step(tokens, targets)
    return dict(s["state"], loss=loss)


def _run_linear(s):
    y = ops.gemm(s["x"], s["w"], residual=s["res"])
    dx = ops.gemm(s["dy"], s["w"], trans_b=True)
    dw = ops.gemm(s["dy"], s["x"], trans_a=True, trans_b=True, out=s["dw"], accumulate=bool(s["accumulate"]))
    return y, dx, dw


def _run_linear_fp8(s):
    wq, ws, wtq, wts = s["w"]
    xq, xs = ops.quant_rows_1x128(s["x"])
    y = ops.gemm_fp8(xq, xs, wq, ws)
    dq, ds = ops.quant_rows_1x128(s["dy"])
    return y, ops.gemm_fp8(dq, ds, wtq, wts)


def _run_experts(s):
    cap, E, k, H, F = s["cap"], s["experts"], s["top_k"], s["hidden"], s["ffn"]
    rows = dict(groups=E, seg_counts=s["live"], seg_rows=cap, seg_mode=1)
    depth = dict(groups=E, seg_counts=s["live"], seg_rows=cap, seg_mode=2, trans_a=True, trans_b=True)
    idx, w, pos, counts = ops.moe_route_fwd(s["logits"], k, cap)
    gu = ops.gemm_grouped(s["xs"], s["wgu"], s["gu"], cap, 2 * F, H, **rows)
    act = ops.swiglu_fwd(gu)
    y = ops.gemm_grouped(act, s["wd"], s["y"], cap, H, F, **rows)
    dact = ops.gemm_grouped(s["dys"], s["wd"], s["dact"], cap, F, H, trans_b=True, **rows)
    dwd = ops.gemm_grouped(s["dys"], act, s["dwd"], H, F, cap, **depth)
    dgu = ops.swiglu_bwd(gu, dact)
    dx = ops.gemm_grouped(dgu, s["wgu"], s["dx"], cap, H, 2 * F, trans_b=True, **rows)
    dwgu = ops.gemm_grouped(dgu, s["xs"], s["dwgu"], 2 * F, H, cap, **depth)
    dlogits = ops.moe_route_bwd(s["logits"], idx, s["dw"], pos)
    return idx, w, pos, counts, y, dx, dwd, dwgu, dlogits


def _run_attention(s):
    B, S, nh, nkv = s["batch"], s["seq"], s["heads"], s["kv_heads"]
    qkv = ops.rope_apply_(s["qkv"], s["table"], S, nh, nkv, 128)
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, 128)
    dqkv = ops.flash_attn_bwd(qkv, out, s["dout"], lse, B, S, nh, nkv, 128)
    ops.rope_apply_(dqkv, s["table"], S, nh, nkv, 128, inverse=True)
    return qkv, out, lse, dqkv


def _run_head(s):
    T = s["rows"]
    y, rstd = ops.rmsnorm_fwd(s["h"], s["gain"])
    logits = ops.gemm(y, s["w"])
    loss = torch.zeros(1, device="cuda")
    dlogits = ops.cross_entropy_(logits, s["targets"], loss, grad_scale=1.0 / T, loss_scale=1.0 / T)
    dy = ops.gemm(dlogits, s["w"], trans_b=True)
    dw = ops.gemm(dlogits, y, trans_a=True, trans_b=True, out_dtype=torch.float32)
    dh, dgain = ops.rmsnorm_bwd(s["h"], s["gain"], rstd, dy)
    return loss, dlogits, dw, dh, dgain


_RUN = dict(step=_run_step, linear=_run_linear, linear_fp8=_run_linear_fp8, experts=_run_experts, attention=_run_attention, head=_run_head)


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------------- what a pass cannot do without
def _step_tokens(c):
    return c["seq_len"] * c["microbatch"] * c["grad_accum"]


def _step_params(c):
    """(parameters, parameters a token multiplies with)."""
    H, F, V = c["hidden_size"], c["ffn_hidden"], c["vocab_size"]
    attn = H * (2 * c["num_heads"] + 2 * c["num_kv_heads"]) * 128
    n = c["num_layers"] * (attn + 3 * H * F + 2 * H) + H + V * H * (1 if c["tie_embeddings"] else 2)
    return n, c["num_layers"] * (attn + 3 * H * F) + V * H


def work(case):
    c = case
    if c["kind"] == "step":
        n, used = _step_params(c)
        T, S = _step_tokens(c), c["seq_len"]
        # forward, input gradients, weight gradients; attention: two products forward, five backward, half of the square
        flops = 6.0 * used * T + 7.0 * T * S * c["num_heads"] * 128 * c["num_layers"]
        # fp32 master, m, v read and written, gradients written, bf16 parameters read and written; tokens and targets
        return {"bytes": 32.0 * n + 8.0 * T, "flops": flops}
    if c["kind"] == "linear":
        M, K, N = c["rows"], c["in_features"], c["out_features"]
        nb = 2.0 * (2 * M * K + 2 * M * N + N * K) + 4.0 * N * K * (2 if c["accumulate"] else 1) + (2.0 * M * N if c["residual"] else 0.0)
        return {"bytes": nb, "flops": 6.0 * M * N * K}
    if c["kind"] == "linear_fp8":
        M, K, N = c["rows"], c["in_features"], c["out_features"]
        return {"bytes": 4.0 * (M * K + M * N) + 2.0 * N * K, "flops": 4.0 * M * N * K}
    if c["kind"] == "experts":
        T, E, k, H, F = c["tokens"], c["experts"], c["top_k"], c["hidden"], c["ffn"]
        # rows of the slabs that hold a token: read x and dy, write y and dx; weights read, their fp32 gradients written; logits
        return {"bytes": 8.0 * T * k * H + (2.0 + 4.0) * 3 * E * H * F + 10.0 * T * E + 16.0 * T * k, "flops": 18.0 * T * k * H * F}
    if c["kind"] == "attention":
        T, nh, nkv = c["batch"] * c["seq"], c["heads"], c["kv_heads"]
        qkv, o = 2.0 * T * (nh + 2 * nkv) * 128, 2.0 * T * nh * 128
        return {"bytes": 3 * qkv + 2 * o + 4.0 * T * nh, "flops": 7.0 * T * c["seq"] * nh * 128}
    T, H, V = c["rows"], c["hidden"], c["vocab"]
    return {"bytes": 2.0 * (2 * T * H + V * H + T * V) + 4.0 * V * H + 8.0 * T, "flops": 6.0 * T * H * V}


def tolerance(case):
    # A step rounds its activations and their gradients to bf16 some twenty times per layer before they meet in a gradient,
    # and the second moment squares it; e4m3 layers turn a last-place change of an activation into a step of an eighth now and
    # then. A single layer's results carry a handful of bf16 roundings.
    if case["kind"] == "step":
        return {"rel": 3e-2 if case["param_dtype"] == "fp8e4m3" else 2e-2}
    return {"rel": 1e-2}

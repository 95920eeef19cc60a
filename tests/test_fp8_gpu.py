"""fp8 (e4m3) block-scaled GEMM and its quantisers against plain PyTorch fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dequant_rows(q, s):
    return q.float() * s.repeat_interleave(128, 1)


def _dequant_blocks(q, s):
    rows, cols = q.shape
    return q.float() * s.repeat_interleave(128, 0)[:rows].repeat_interleave(128, 1)[:, :cols]


def test_quantisers_round_trip():
    from cai_b200 import ops
    torch.manual_seed(0)
    x = (torch.randn(300, 512, device="cuda") * torch.rand(300, 1, device="cuda") * 8).to(torch.bfloat16)
    q, s = ops.quant_rows_1x128(x)
    amax = x.float().view(300, 4, 128).abs().amax(-1)
    assert torch.allclose(s, amax / 448, rtol=1e-6)
    back = _dequant_rows(q, s)
    assert ((back - x.float()).abs() <= 0.07 * amax.repeat_interleave(128, 1) + 1e-6).all()   # e4m3: 3 mantissa bits
    w = torch.randn(384, 200, device="cuda").to(torch.bfloat16)
    qw, sw, qt, st = ops.quant_blocks_128x128(w, transposed=True)
    assert sw.shape == (3, 2) and st.shape == (2, 3) and torch.equal(st, sw.t().contiguous())
    assert torch.equal(qt.view(torch.uint8), qw.view(torch.uint8).t().contiguous())
    backw = _dequant_blocks(qw, sw)
    assert (backw - w.float()).abs().max() <= 0.07 * w.float().abs().max()


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (256, 512, 1024), (200, 264, 384), (1024, 4096, 2048)])
def test_gemm_matches_dequantised_reference(M, N, K):
    from cai_b200 import ops
    torch.manual_seed(1)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    xq, sx = ops.quant_rows_1x128(x)
    wq, sw = ops.quant_blocks_128x128(w)
    ref = _dequant_rows(xq, sx) @ _dequant_blocks(wq, sw).t()     # exactly what the kernel computes, in fp32
    out32 = ops.gemm_fp8(xq, sx, wq, sw, out_dtype=torch.float32)
    assert torch.allclose(out32, ref, atol=1e-3 * ref.abs().max().item(), rtol=1e-3)
    res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    out16 = ops.gemm_fp8(xq, sx, wq, sw, residual=res)
    assert torch.allclose(out16.float(), ref + res.float(), atol=2e-2 * ref.abs().max().item(), rtol=2e-2)
    # against the unquantised product the error is the e4m3 rounding of both operands
    full = x.float() @ w.float().t()
    rel = ((out32 - full).norm() / full.norm()).item()
    assert rel < 0.08, rel
    from cai_b200.ops import _lib
    assert _lib.device_status(clear=True) == 0


def test_training_with_fp8_linear_layers_tracks_bf16():
    """param_dtype = fp8e4m3: forward and input-gradient GEMMs of the linear layers run in e4m3 with
    block scales. The loss curve must stay within a few percent of the bf16 run and fall the same way."""
    from pathlib import Path
    from cai_b200.runtime.engine import Engine, synthetic_batch
    text = (Path(__file__).resolve().parent.parent / "configs" / "tiny.cfg").read_text()
    curves = {}
    for dt in ("bf16", "fp8e4m3"):
        eng = Engine(config_text=text.replace("param_dtype   = bf16", f"param_dtype   = {dt}"), rank=0, world=1, local_rank=0)
        m = eng.model
        rows = eng.hdr.num_microbatches * m.microbatch
        tok, tgt = synthetic_batch(m.vocab_size, m.seq_len, rows, step=0, seed=9)
        curves[dt] = [eng.step(tok, tgt) for _ in range(8)]
        kernels = {int(x.kernel) for x in eng.plan.exec}
        eng.close()
        if dt == "fp8e4m3":
            from cai_b200 import plan as planlib
            assert planlib.K_GEMM_FP8 in kernels and planlib.K_QUANT_FP8 in kernels
    a, b = curves["bf16"], curves["fp8e4m3"]
    assert b[-1] < b[0] - 0.3, b
    for x, y in zip(a, b):
        assert abs(x - y) < 0.03 * max(1.0, x), (a, b)


def _strided(t, pad):
    big = torch.zeros(t.shape[0], t.shape[1] + pad, device=t.device, dtype=t.dtype)
    big[:, :t.shape[1]] = t
    return big


# The quantisers' wide form (16-byte pieces) against their narrow one, which takes rows at odd pitches: the same bytes.
@pytest.mark.parametrize("rows,cols", [(1, 128), (63, 384), (65, 128), (300, 1152)])
def test_quant_rows_forms_agree(rows, cols):
    import ctypes
    from cai_b200 import ops
    torch.manual_seed(4)
    x = (torch.randn(rows, cols, device="cuda") * 3).to(torch.bfloat16)
    x[rows // 2, :128] = 0
    q, s = ops.quant_rows_1x128(x)
    xp = _strided(x, 4)
    q2, s2 = torch.zeros_like(q), torch.zeros_like(s)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert ops.lib().cai_quant_rows_1x128(p(xp), ctypes.c_longlong(cols + 4), p(q2), ctypes.c_longlong(cols), p(s2), rows, cols,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert torch.equal(q.view(torch.uint8), q2.view(torch.uint8)) and torch.equal(s, s2)


@pytest.mark.parametrize("rows,cols", [(16, 8), (128, 128), (144, 392), (400, 264)])
def test_quant_blocks_forms_agree(rows, cols):
    import ctypes
    from cai_b200 import ops
    torch.manual_seed(5)
    w = torch.randn(rows, cols, device="cuda").to(torch.bfloat16)
    q, s, qt, st = ops.quant_blocks_128x128(w, transposed=True)
    wp = _strided(w, 3)
    q2, s2, qt2, st2 = torch.zeros_like(q), torch.zeros_like(s), torch.zeros_like(qt), torch.zeros_like(st)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    n = ctypes.c_longlong
    assert ops.lib().cai_quant_blocks_128x128(p(wp), n(cols + 3), p(q2), n(q.stride(0)), p(qt2), n(qt.stride(0)), p(s2), p(st2), rows, cols,
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    for a, b in ((q, q2), (qt, qt2)):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    assert torch.equal(s, s2) and torch.equal(st, st2)


# one row, halves of the 256-row pair tile, one past a tile; a fraction of a column tile; one k-block, and one past the eight whose scales
# come in together; several tiles per pair. In float64 from the quantised operands.
@pytest.mark.parametrize("M,N,K", [(1, 8, 128), (127, 136, 256), (129, 264, 1152), (257, 640, 1024), (300, 72, 2176), (2300, 4104, 640)])
def test_gemm_edges(M, N, K):
    from cai_b200 import ops
    torch.manual_seed(M)
    xq, sx = ops.quant_rows_1x128(torch.randn(M, K, device="cuda").to(torch.bfloat16))
    wq, sw = ops.quant_blocks_128x128((torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16))
    A, B = _dequant_rows(xq, sx).double(), _dequant_blocks(wq, sw).double()
    ref = A @ B.t()
    bound = K * 2.0 ** -23 * (A.abs() @ B.abs().t())       # products of e4m3 are exact; sums and scalings in fp32
    wide = torch.full((M, N + 16), 7.0, device="cuda")
    ops.gemm_fp8(xq, sx, wq, sw, out=wide[:, :N])
    assert ((wide[:, :N] - ref).abs() <= bound).all() and bool((wide[:, N:] == 7.0).all())
    res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    out = ops.gemm_fp8(xq, sx, wq, sw, residual=res)
    want = ref + res.double()
    assert ((out.double() - want).abs() <= bound + 2.0 ** -8 * want.abs() + 1e-6).all()


def test_one_cta_and_pair_forms_give_the_same_bits():
    from cai_b200 import ops
    torch.manual_seed(0)
    K, N = 1152, 28672                                     # 128 rows run on one CTA per tile, 256 rows on pairs
    xq, sx = ops.quant_rows_1x128(torch.randn(256, K, device="cuda").to(torch.bfloat16))
    wq, sw = ops.quant_blocks_128x128((torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16))
    both = ops.gemm_fp8(xq, sx, wq, sw, out_dtype=torch.float32)
    half = ops.gemm_fp8(xq[:128], sx[:128].contiguous(), wq, sw, out_dtype=torch.float32)
    assert torch.equal(both[:128], half)


# k-blocks around the scales' groups of four and eight, odd and even (the TMEM buffer a tile starts in), more tiles than CTA pairs, ragged edges.
@pytest.mark.parametrize("kb", [1, 2, 3, 4, 5, 7, 8, 9, 13, 17])
@pytest.mark.parametrize("M,N", [(2304, 2304), (300, 1000)])
def test_pair_form_k_blocks(M, N, kb):
    from cai_b200 import ops
    torch.manual_seed(kb)
    x = torch.randn(M, kb * 128, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, kb * 128, device="cuda") * 0.05).to(torch.bfloat16)
    (xq, sx), (wq, sw) = ops.quant_rows_1x128(x), ops.quant_blocks_128x128(w)
    a, b = _dequant_rows(xq, sx).double(), _dequant_blocks(wq, sw).double()
    out = ops.gemm_fp8(xq, sx, wq, sw, out_dtype=torch.float32)
    # products of e4m3 are exact in fp32; K sums and a scaling per k-block, each off by at most 2^-24 of what it adds up to (the tensor
    # core's sums within a k-block may be truncated to 2^-13 of their largest term, as they are in every product of this format)
    bound = (2.0 ** -13 + (128 + 3 * kb) * 2.0 ** -24) * (a.abs() @ b.abs().t()) + 1e-9
    assert ((out.double() - a @ b.t()).abs() <= bound).all()
    assert ops.device_status() == 0

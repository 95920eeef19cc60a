"""Flash attention (forward and backward) against a plain PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref_attention(qkv, B, S, nh, nkv, hd):
    x = qkv.float().view(B, S, nh + 2 * nkv, hd)
    q = x[:, :, :nh].transpose(1, 2)                       # B nh S hd
    k = x[:, :, nh:nh + nkv].transpose(1, 2)
    v = x[:, :, nh + nkv:].transpose(1, 2)
    rep = nh // nkv
    k = k.repeat_interleave(rep, dim=1)
    v = v.repeat_interleave(rep, dim=1)
    s = (q @ k.transpose(-1, -2)) * hd ** -0.5
    mask = torch.ones(S, S, device=qkv.device, dtype=torch.bool).tril()
    s = s.masked_fill(~mask, float("-inf"))
    lse = torch.logsumexp(s, -1)
    o = torch.softmax(s, -1) @ v
    return o.transpose(1, 2).reshape(B * S, nh * hd), lse


@pytest.mark.parametrize("B,S,nh,nkv", [(1, 128, 2, 2), (2, 256, 4, 2), (1, 384, 4, 1), (1, 1024, 8, 2),
                                        (2, 2048, 4, 4), (1, 4096, 16, 8)])
@pytest.mark.parametrize("variant", [1, 2])
def test_flash_attn_fwd(B, S, nh, nkv, variant):
    from cai_b200 import ops
    torch.manual_seed(0)
    hd = 128
    qkv = torch.randn(B * S, (nh + 2 * nkv) * hd, device="cuda").to(torch.bfloat16)
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, hd, variant=variant)
    ref, lse_ref = _ref_attention(qkv, B, S, nh, nkv, hd)
    rel = ((out.float() - ref).norm() / ref.norm()).item()
    assert rel < 1e-2, rel
    assert (out.float() - ref).abs().max().item() < 6e-2
    assert torch.allclose(lse, lse_ref, atol=2e-2, rtol=1e-3)


# The dK / dV kernel has two forms: one CTA per kv group looping over the group's query heads (grids that fill
# the GPU: B * kv groups * key tiles >= SM count) and one CTA per query head with chained adds (small grids).
# (1, 4096, 16, 8) is the shape of the headline model on one GPU and takes the first form with two heads per
# group; (1, 512, 8, 1) chains eight heads; (2, 4096, 2, 1) is the tp = 8 shape with two microbatches per launch.
@pytest.mark.parametrize("B,S,nh,nkv", [(1, 128, 2, 2), (2, 256, 4, 2), (1, 384, 4, 1), (1, 1024, 8, 2),
                                        (1, 4096, 16, 8), (1, 512, 8, 1), (2, 4096, 2, 1)])
def test_flash_attn_bwd(B, S, nh, nkv):
    from cai_b200 import ops
    if not hasattr(ops.lib(), "cai_flash_attn_bwd"):
        pytest.skip("backward kernel not built")
    torch.manual_seed(1)
    hd = 128
    qkv = torch.randn(B * S, (nh + 2 * nkv) * hd, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B * S, nh * hd, device="cuda").to(torch.bfloat16)
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, hd)
    dqkv = ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, hd)
    x = qkv.float().requires_grad_(True)
    ref, _ = _ref_attention(x, B, S, nh, nkv, hd)
    ref.backward(dout.float())
    g = x.grad.view(B * S, nh + 2 * nkv, hd)
    d = dqkv.float().view(B * S, nh + 2 * nkv, hd)
    for name, sl in (("dq", slice(0, nh)), ("dk", slice(nh, nh + nkv)), ("dv", slice(nh + nkv, nh + 2 * nkv))):
        rel = ((d[:, sl] - g[:, sl]).norm() / g[:, sl].norm()).item()
        assert rel < 2e-2, (name, rel)


# The operand rings of the backward kernels turn over after 1, 2 and 3 tiles: sequences of one to seven tiles, one and
# several heads per group in both forms of the dK / dV kernel (one head per CTA where everything is resident at once, a sweep
# over the group where the grid fills the GPU), and the same bits in every run.
@pytest.mark.parametrize("B,S,nh,nkv", [(1, 128, 1, 1), (1, 256, 3, 1), (3, 384, 9, 3), (1, 896, 4, 4), (40, 512, 3, 1)])
def test_flash_attn_bwd_rings(B, S, nh, nkv):
    from cai_b200 import ops
    torch.manual_seed(2)
    hd = 128
    qkv = torch.randn(B * S, (nh + 2 * nkv) * hd, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B * S, nh * hd, device="cuda").to(torch.bfloat16)
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, hd)
    dqkv = ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, hd)
    again = ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, hd)
    assert torch.equal(dqkv, again)
    x = qkv.float().requires_grad_(True)
    ref, _ = _ref_attention(x, B, S, nh, nkv, hd)
    ref.backward(dout.float())
    # P, dS and the results are rounded to bf16 (2^-9 relative each, independent): well under 1e-2 in the 2-norm
    rel = ((dqkv.float() - x.grad).norm() / x.grad.norm()).item()
    assert rel < 1e-2, rel


def test_flash_attn_bwd_takes_an_output_on_eight_bytes():
    """The row sums of dO * O read O in 16-byte pieces where it lies on 16 bytes and in 8-byte pieces where it does not: the same bits."""
    from cai_b200 import ops
    torch.manual_seed(3)
    B, S, nh, nkv, hd = 3, 384, 3, 1, 128
    qkv = torch.randn(B * S, (nh + 2 * nkv) * hd, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B * S, nh * hd, device="cuda").to(torch.bfloat16)
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, hd)
    room = torch.empty(out.numel() + 4, device="cuda", dtype=torch.bfloat16)
    moved = room[4:].view_as(out).copy_(out)
    assert moved.data_ptr() % 16 == 8
    d = [torch.empty(B, nh, S, device="cuda") for _ in range(2)]
    got = [ops.flash_attn_bwd(qkv, o, dout, lse, B, S, nh, nkv, hd, delta=x) for o, x in zip((out, moved), d)]
    assert torch.equal(d[0], d[1]) and torch.equal(got[0], got[1])
    want = (dout.float() * out.float()).view(B, S, nh, hd).sum(-1).transpose(1, 2)
    assert ((d[0] - want).abs() <= 2.0 ** -23 * 128 * (dout.float() * out.float()).abs().view(B, S, nh, hd).sum(-1).transpose(1, 2)).all()


# one key block and several, an odd number of tiles, grouped heads; more CTAs than two per SM
@pytest.mark.parametrize("B,S,nh,nkv", [(1, 128, 1, 1), (3, 384, 6, 2), (8, 640, 9, 3), (2, 1152, 16, 8), (1, 4224, 2, 1)])
def test_forward_forms_give_the_same_bits(B, S, nh, nkv):
    from cai_b200 import ops
    torch.manual_seed(S)
    qkv = (torch.randn(B * S, (nh + 2 * nkv) * 128, device="cuda") * 2).to(torch.bfloat16)   # the running maximum moves now and then
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, 128, variant=2)
    for variant in (0, 1, 3):
        o, l = ops.flash_attn_fwd(qkv, B, S, nh, nkv, 128, variant=variant)
        assert torch.equal(o, out) and torch.equal(l, lse)


# dK / dV and dQ in one launch against each by itself: the same CTAs, so the same bits. Grids of one CTA each, smaller and larger than the GPU, split
# heads (the first three with several query heads per kv head) and not.
@pytest.mark.parametrize("B,S,nh,nkv", [(1, 128, 1, 1), (1, 128, 4, 1), (2, 384, 6, 2), (1, 512, 8, 1), (8, 384, 12, 4), (3, 640, 9, 3), (1, 2048, 16, 8)])
def test_flash_attn_bwd_parts_together(B, S, nh, nkv):
    from cai_b200 import ops
    torch.manual_seed(2)
    qkv = torch.randn(B * S, (nh + 2 * nkv) * 128, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B * S, nh * 128, device="cuda").to(torch.bfloat16)
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, 128)
    delta = torch.empty((B, nh, S), device="cuda")
    whole = ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, 128, delta=delta)
    parts, kv_only, q_only = (torch.full_like(qkv, 7.0) for _ in range(3))
    for p in (1, 4, 2):
        ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, 128, dqkv=parts, delta=torch.empty_like(delta) if p == 1 else delta, parts=p)
    ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, 128, dqkv=kv_only, delta=delta, parts=2)
    ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, 128, dqkv=q_only, delta=delta, parts=4)
    assert torch.equal(whole, parts)
    q = nh * 128
    assert torch.equal(whole[:, :q], q_only[:, :q]) and bool((q_only[:, q:] == 7.0).all())
    assert torch.equal(whole[:, q:], kv_only[:, q:]) and bool((kv_only[:, :q] == 7.0).all())


# The backward with the inverse rotary embedding of dQ and dK in it against the two passes: the same bits. Chained heads and not.
@pytest.mark.parametrize("B,S,nh,nkv", [(1, 128, 1, 1), (4, 128, 2, 1), (1, 512, 8, 1), (3, 640, 9, 3), (2, 1024, 16, 8)])
@pytest.mark.parametrize("parts", [7, 4, 2])
def test_flash_attn_bwd_rotated_back(B, S, nh, nkv, parts):
    import ctypes
    from cai_b200 import ops
    torch.manual_seed(3)
    qkv = torch.randn(B * S, (nh + 2 * nkv) * 128, device="cuda").to(torch.bfloat16)
    dout = torch.randn(B * S, nh * 128, device="cuda").to(torch.bfloat16)
    table = ops.rope_table(S, 128)
    out, lse = ops.flash_attn_fwd(qkv, B, S, nh, nkv, 128)
    delta = torch.empty((B, nh, S), device="cuda")
    want = torch.zeros_like(qkv)
    ops.flash_attn_bwd(qkv, out, dout, lse, B, S, nh, nkv, 128, dqkv=want, delta=delta)
    ops.rope_apply_(want, table, S, nh, nkv, 128, inverse=True)
    got = torch.zeros_like(qkv)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (qkv, out, dout, lse, delta, got, table)]
    rc = ops.lib().cai_flash_attn_bwd_rope(*p, B, S, nh, nkv, 128, ctypes.c_float(128 ** -0.5), parts, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and ops.device_status() == 0
    q = nh * 128
    if parts & 4:
        assert torch.equal(got[:, :q], want[:, :q])
    if parts & 2:
        assert torch.equal(got[:, q:], want[:, q:])
    assert bool((got[:, :q] == 0).all()) == (not parts & 4) and bool((got[:, q:] == 0).all()) == (not parts & 2)

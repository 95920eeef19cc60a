"""GEMM on CTA pairs and its split along K: edges of the 256 x 256 / 256 x 128 tiles, of a stage and of the K slices."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# M, N, K: one row, half tiles, one past a tile, K of a fraction of a block, of an odd number of blocks, fewer slices than
# blocks; few tiles (split), one wave and several waves of tiles (persistent)
SHAPES = [(1, 8, 8), (128, 128, 64), (129, 136, 72), (256, 256, 128), (257, 264, 1000), (333, 1024, 3000), (40, 3000, 512),
          (1000, 1152, 3840), (513, 120, 4104), (4096, 5000, 200), (2500, 4104, 136)]


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_pair_gemm_edges(M, N, K, ta, tb):
    from cai_b200 import ops
    torch.manual_seed(0)
    M = (M + 7) // 8 * 8 if ta else M                      # a contiguous M has to be a multiple of 8
    a = torch.randn((K, M) if ta else (M, K), device="cuda").to(torch.bfloat16)
    b = torch.randn((K, N) if tb else (N, K), device="cuda").to(torch.bfloat16)
    A, B = (a.t() if ta else a).float(), (b if tb else b.t()).float()
    ref = A @ B
    # products of bf16 are exact in fp32; two sums of K terms in different orders differ by at most 2 K 2^-24 sum |a b|
    bound = 2 * K * 2.0 ** -24 * (A.abs() @ B.abs()) + 1e-6
    out = torch.full((M, N), 2.0, device="cuda")
    ops.gemm(a, b, trans_a=ta, trans_b=tb, out=out, accumulate=True, alpha=0.5)
    assert ((out - (2.0 + 0.5 * ref)).abs() <= bound + 2.0 ** -23 * (2.0 + ref.abs())).all()
    wide = torch.full((M, N + 16), 7.0, device="cuda")     # a pitch wider than the row: nothing outside may be touched
    ops.gemm(a, b, trans_a=ta, trans_b=tb, out=wide[:, :N])
    assert ((wide[:, :N] - ref).abs() <= bound).all() and bool((wide[:, N:] == 7.0).all())
    res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    c = ops.gemm(a, b, trans_a=ta, trans_b=tb, residual=res)
    want = ref + res.float()
    assert ((c.float() - want).abs() <= bound + 2.0 ** -8 * want.abs() + 1e-6).all()    # and one rounding to bf16
    assert torch.equal(c, ops.gemm(a, b, trans_a=ta, trans_b=tb, residual=res))         # the order of summation is fixed
    from cai_b200.ops import _lib
    assert _lib.device_status(clear=True) == 0


@pytest.mark.parametrize("M,N", [(200, 72), (256, 136), (130, 256)])
def test_pair_gemm_groups_do_not_touch_each_other(M, N):
    """Group sizes that are no multiple of a tile or of the 32-row boxes: rows past a group belong to the next one."""
    from cai_b200 import ops
    torch.manual_seed(1)
    G, K = 3, 192
    a = torch.randn(G * M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(G * N, K, device="cuda").to(torch.bfloat16)
    out = torch.zeros(G * M, N, device="cuda")
    ops.gemm_grouped(a, b, out, M, N, K, groups=G)
    for g in range(G):
        A, B = a[g * M:(g + 1) * M].float(), b[g * N:(g + 1) * N].float()
        assert ((out[g * M:(g + 1) * M] - A @ B.t()).abs() <= 2 * K * 2.0 ** -24 * (A.abs() @ B.abs().t()) + 1e-6).all()


# Split along K, where a CTA of the cluster has no rows (M of at most half a tile, or half a tile past a whole one) and where the last
# slab of columns lies partly or wholly past N. Launched back to back, so that a CTA that left early would meet its successor.
@pytest.mark.parametrize("M,N,K", [(8, 8, 512), (128, 136, 1024), (129, 264, 4096), (264, 104, 8192), (384, 1000, 3000), (130, 1032, 264)])
def test_split_gemm_empty_halves(M, N, K):
    from cai_b200 import ops
    from cai_b200.ops import _lib
    torch.manual_seed(3)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    bound = 2 * K * 2.0 ** -24 * (a.float().abs() @ b.float().abs().t()) + 1e-6    # two sums of K exact products in fp32
    outs = [ops.gemm(a, b, out_dtype=torch.float32) for _ in range(50)]
    assert ((outs[0] - a.float() @ b.float().t()).abs() <= bound).all()
    assert all(torch.equal(outs[0], o) for o in outs[1:])
    assert _lib.device_status(clear=True) == 0


# The even CTA's last commit arrives on both CTAs of a pair; the one without rows has to have seen it before it ends. Two streams, so that
# the SMs of an early leaver would be handed to the other stream's clusters at once.
def test_split_gemm_empty_halves_on_two_streams():
    from cai_b200 import ops
    from cai_b200.ops import _lib
    torch.manual_seed(4)
    cases = []
    for M, N, K in ((8, 1024, 2048), (136, 520, 4096)):
        a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
        b = torch.randn(N, K, device="cuda").to(torch.bfloat16)
        bound = 2 * K * 2.0 ** -24 * (a.float().abs() @ b.float().abs().t()) + 1e-6
        cases.append((a, b, a.float() @ b.float().t(), bound, torch.cuda.Stream()))
    torch.cuda.synchronize()
    outs = [[] for _ in cases]
    for _ in range(30):
        for o, (a, b, _, _, st) in zip(outs, cases):
            with torch.cuda.stream(st):
                o.append(ops.gemm(a, b, out_dtype=torch.float32))
    torch.cuda.synchronize()
    for o, (_, _, ref, bound, _) in zip(outs, cases):
        assert all(((v - ref).abs() <= bound).all() for v in o)
    assert _lib.device_status(clear=True) == 0


# A last tile's accumulator is handed back to the even CTA with nobody waiting for it: short kernels back to back on two streams, one tile
# per pair, both widths, so that a pair that parted early would be replaced at once.
def test_pair_gemm_short_kernels_on_two_streams():
    from cai_b200 import ops
    from cai_b200.ops import _lib
    torch.manual_seed(5)
    cases = []
    for M, N, K in ((2000, 2000, 64), (2304, 4104, 72)):
        a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
        b = torch.randn(N, K, device="cuda").to(torch.bfloat16)
        bound = 2 * K * 2.0 ** -24 * (a.float().abs() @ b.float().abs().t()) + 1e-6
        cases.append((a, b, a.float() @ b.float().t(), bound, torch.cuda.Stream()))
    torch.cuda.synchronize()
    outs = [[] for _ in cases]
    for _ in range(20):
        for o, (a, b, _, _, st) in zip(outs, cases):
            with torch.cuda.stream(st):
                o.append(ops.gemm(a, b, out_dtype=torch.float32))
    torch.cuda.synchronize()
    for o, (_, _, ref, bound, _) in zip(outs, cases):
        assert all(((v - ref).abs() <= bound).all() for v in o)
    assert _lib.device_status(clear=True) == 0


# A limit on the SMs in every form: persistent wide and narrow, two and four slices (in turns of several launches): the same bits, with
# every epilogue, and the ragged last turn.
@pytest.mark.parametrize("M,N,K", [(4096, 4104, 264), (1536, 1536, 520), (333, 1024, 3000), (300, 968, 2048)])
def test_pair_gemm_under_a_limit(M, N, K):
    from cai_b200 import ops
    from cai_b200.ops import _lib
    torch.manual_seed(6)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    old = torch.randn(M, N, device="cuda")
    want = ops.gemm(a, b, out_dtype=torch.float32), ops.gemm(a, b, residual=res), ops.gemm(a, b, out=old.clone(), accumulate=True)
    for limit in (1, 2, 10, 60, 147):
        got = (ops.gemm(a, b, out_dtype=torch.float32, sm_limit=limit), ops.gemm(a, b, residual=res, sm_limit=limit),
               ops.gemm(a, b, out=old.clone(), accumulate=True, sm_limit=limit))
        assert all(torch.equal(x, y) for x, y in zip(got, want)), limit
    assert _lib.device_status(clear=True) == 0


FORMS = [(4096, 4104, 264), (1536, 1536, 520), (336, 1024, 3000), (256, 1920, 2048)]     # 256-wide, 128-wide, two and four slices


def _padded(rows, cols, pad, value=7.0, dtype=torch.bfloat16):
    """A random matrix as the left part of rows that are `pad` wider, and the whole."""
    whole = torch.full((rows, cols + pad), value, device="cuda", dtype=dtype)
    whole[:, :cols] = torch.randn(rows, cols, device="cuda").to(dtype)
    return whole[:, :cols], whole


# Pitches wider than the row for every operand, and the residual read in place of the result: the bits of the plain call, and nothing
# touched beside the rows.
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True)])
@pytest.mark.parametrize("M,N,K", FORMS)
def test_pair_gemm_pitches_and_residual_in_place(M, N, K, ta, tb):
    from cai_b200 import ops
    torch.manual_seed(8)
    a, _ = _padded(*((K, M) if ta else (M, K)), 16)
    b, _ = _padded(*((K, N) if tb else (N, K)), 24)
    res, res_whole = _padded(M, N, 40)
    kw = dict(trans_a=ta, trans_b=tb)
    want = ops.gemm(a.contiguous(), b.contiguous(), residual=res.contiguous(), **kw)
    assert torch.equal(ops.gemm(a, b, residual=res, **kw), want)
    ref = ((a.t() if ta else a).float() @ (b if tb else b.t()).float()) + res.float()
    bound = 2 * K * 2.0 ** -24 * ((a.t() if ta else a).float().abs() @ (b if tb else b.t()).float().abs()) + 2.0 ** -8 * ref.abs() + 1e-6
    assert ((want.float() - ref).abs() <= bound).all()       # two sums of K exact products, one rounding to bf16
    out, out_whole = _padded(M, N, 8)
    ops.gemm(a, b, residual=res, out=out, **kw)
    assert torch.equal(out, want) and bool((out_whole[:, N:] == 7.0).all())
    ops.gemm(a, b, residual=res, out=res, **kw)
    assert torch.equal(res, want) and bool((res_whole[:, N:] == 7.0).all())
    acc, acc_whole = _padded(M, N, 4, dtype=torch.float32)
    want32 = ops.gemm(a.contiguous(), b.contiguous(), out=acc.contiguous(), accumulate=True, **kw)
    ops.gemm(a, b, out=acc, accumulate=True, **kw)
    assert torch.equal(acc, want32) and bool((acc_whole[:, N:] == 7.0).all())


# Adding to gradients below 2^-126: the persistent forms add in L2, the split form in registers; neither flushes. All values exact.
@pytest.mark.parametrize("M,N,K", [(4096, 4104, 64), (256, 128, 64), (336, 1024, 3000)])
def test_accumulation_keeps_subnormals(M, N, K):
    from cai_b200 import ops
    a = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.zeros(N, K, device="cuda", dtype=torch.bfloat16)
    a[:, 0], b[:, 0] = 2.0 ** -100, 2.0 ** -30
    for old in (0.0, 2.0 ** -130, 2.0 ** -140, -2.0 ** -126):
        out = torch.full((M, N), old, device="cuda")
        ops.gemm(a, b, out=out, accumulate=True)
        assert bool((out.double() == old + 2.0 ** -130).all()), old


def _ragged_counts(kind, slabs, seg_rows, g):
    edges = [0, 1, 63, 64, 65, 127, 128, 129, 191, 192, 255, 256, 257, seg_rows - 1, seg_rows, seg_rows + 5]
    if kind == "edges":
        return torch.tensor([edges[i % len(edges)] for i in range(slabs)], dtype=torch.int32)
    if kind == "one":
        c = torch.zeros(slabs, dtype=torch.int32)
        c[slabs // 2] = seg_rows
        return c
    if kind == "none":
        return torch.zeros(slabs, dtype=torch.int32)
    return torch.randint(0, seg_rows + 1, (slabs,), generator=g, dtype=torch.int32)


# Live halves counted ahead (up to 256 slabs) and the walk over all tiles (beyond): one slab and several per group, few groups and more than a
# warp has lanes, slabs of an odd number of 128-row halves (a tile takes halves of two slabs), more row tiles than a raster group of eight.
@pytest.mark.parametrize("groups,per_group,seg_rows,N,K", [(16, 1, 128, 256, 128), (5, 3, 384, 264, 192), (4, 4, 256, 512, 64),
                                                           (2, 2, 2432, 384, 256), (300, 1, 128, 128, 64), (100, 3, 128, 72, 64), (256, 1, 128, 136, 64),
                                                           (40, 3, 384, 136, 64), (85, 3, 128, 72, 64), (1, 256, 128, 72, 64)])
@pytest.mark.parametrize("kind", ["edges", "random", "one", "none"])
def test_grouped_ragged_rows(groups, per_group, seg_rows, N, K, kind):
    from cai_b200 import ops
    g = torch.Generator().manual_seed(groups * 7 + seg_rows)
    M = per_group * seg_rows
    counts = _ragged_counts(kind, groups * per_group, seg_rows, g)
    a = (torch.randn(groups * M, K, generator=g) * 0.5).bfloat16().cuda()
    b = (torch.randn(groups * N, K, generator=g) * 0.5).bfloat16().cuda()
    out = torch.full((groups * M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_grouped(a, b, out, M, N, K, groups=groups, seg_counts=counts.cuda(), seg_rows=seg_rows, seg_mode=1)
    A, B = a.view(groups, M, K).double(), b.view(groups, N, K).double()
    ref = torch.einsum("gmk,gnk->gmn", A, B).view(-1, seg_rows, N)
    # one rounding to bf16, and a sum of K exact products in fp32
    bound = 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * torch.einsum("gmk,gnk->gmn", A.abs(), B.abs()).view(-1, seg_rows, N)
    got = out.view(-1, seg_rows, N).double()
    for s, c in enumerate(counts.tolist()):
        c = min(c, seg_rows)
        whole = (c + 127) // 128 * 128           # halves of 128 rows are written whole
        assert ((got[s, :c] - ref[s, :c]).abs() <= bound[s, :c]).all()
        assert bool((got[s, whole:] == 7.0).all())


@pytest.mark.parametrize("groups,per_group,seg_rows,M,N", [(8, 1, 256, 256, 128), (3, 3, 384, 264, 136), (2, 5, 128, 128, 512)])
@pytest.mark.parametrize("kind", ["edges", "random", "one", "none"])
@pytest.mark.parametrize("accumulate", [False, True])
def test_grouped_ragged_depth(groups, per_group, seg_rows, M, N, kind, accumulate):
    from cai_b200 import ops
    g = torch.Generator().manual_seed(groups * 5 + seg_rows)
    K = per_group * seg_rows
    counts = _ragged_counts(kind, groups * per_group, seg_rows, g)
    a = (torch.randn(groups * K, M, generator=g) * 0.5).bfloat16()
    b = (torch.randn(groups * K, N, generator=g) * 0.5).bfloat16()
    # rows past a count up to the end of its 64-row block are zero, as a dispatch leaves them; later ones are never read
    for s, c in enumerate(counts.tolist()):
        c = min(c, seg_rows)
        end = (c + 63) // 64 * 64
        for t in (a, b):
            t[s * seg_rows + c:s * seg_rows + end] = 0
            t[s * seg_rows + end:(s + 1) * seg_rows] = float("nan")
    out = torch.full((groups * M, N), 3.0, device="cuda")
    ops.gemm_grouped(a.cuda(), b.cuda(), out, M, N, K, groups=groups, trans_a=True, trans_b=True, accumulate=accumulate,
                     seg_counts=counts.cuda(), seg_rows=seg_rows, seg_mode=2)
    A, B = a.view(groups, K, M).nan_to_num().double(), b.view(groups, K, N).nan_to_num().double()
    ref = torch.einsum("gkm,gkn->gmn", A, B).reshape(-1, N) + (3.0 if accumulate else 0.0)
    bound = (K + 1) * 2.0 ** -24 * (torch.einsum("gkm,gkn->gmn", A.abs(), B.abs()).reshape(-1, N) + 3.0)
    assert ((out.cpu().double() - ref).abs() <= bound).all()


# Full slabs of an odd number of 128-row halves cost what the same rows without slabs cost: two neighbouring halves share a tile, of
# whatever slabs they are. (With tiles that end at their slab these take 1.7 and 1.4 times as long.)
@pytest.mark.parametrize("groups,per,seg_rows", [(1, 8, 128), (8, 8, 384)])
def test_full_slabs_cost_what_plain_rows_cost(groups, per, seg_rows):
    from cai_b200 import ops
    M, N, K = per * seg_rows, 3072, 4096
    a = torch.randn(groups * M, K, device="cuda").bfloat16()
    b = torch.randn(groups * N, K, device="cuda").bfloat16()
    out = torch.empty(groups * M, N, device="cuda", dtype=torch.bfloat16)
    counts = torch.full((groups * per,), seg_rows, device="cuda", dtype=torch.int32)

    times = {True: [], False: []}
    for i in range(20):                  # in turn, so that a change of clock meets both
        ragged = dict(seg_counts=counts, seg_rows=seg_rows, seg_mode=1) if i % 2 else {}
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(100000)
        s.record()
        ops.gemm_grouped(a, b, out, M, N, K, groups=groups, **ragged)
        e.record()
        torch.cuda.synchronize()
        times[bool(ragged)].append(s.elapsed_time(e))
    # both run with 256-row tiles along the whole of K; the plain one in the form that its shape asks for
    assert sorted(times[True])[4] < 1.25 * sorted(times[False])[4]


def _call(x, w, dy, dw=None, accumulate=False, residual=None):
    """A linear layer's input gradient (dw None) or weight gradient, as a call and as a function that runs it by itself."""
    from cai_b200 import ops
    from cai_b200.ops import _lib
    if dw is None:
        out = torch.full_like(x, 3.0)
        a, b, (M, K), N, ta, tb, epi = dy, w, dy.shape, w.shape[1], 0, 1, 3 if residual is not None else 0
    else:
        out = dw.clone()
        a, b, (K, M), N, ta, tb, epi = dy, x, dy.shape, x.shape[1], 1, 1, 2 if accumulate else 1
    call = _lib.GemmCall(A=a.data_ptr(), B=b.data_ptr(), C=out.data_ptr(), R=residual.data_ptr() if residual is not None else None, lda=a.stride(0),
                         ldb=b.stride(0), ldc=out.stride(0), ldr=residual.stride(0) if residual is not None else 0, M=M, N=N, K=K, a_mn_major=ta,
                         b_mn_major=tb, epi=epi, alpha=1.0)
    alone = dw.clone() if dw is not None else torch.full_like(x, 3.0)
    ops.gemm(a, b, trans_a=bool(ta), trans_b=bool(tb), out=alone, accumulate=bool(epi == 2), residual=residual)
    return call, out, alone


# Both gradients of a linear layer in one launch against one launch each, and in either order: the same bits. Tokens, in and out features: persistent
# tiles of 256 and of 128 columns; clusters of four slices and of two, of forms that differ (one sum beside a split one, two slices beside four),
# with pairs and clusters that are left without a tile; one row, ragged edges; three that stay two launches.
@pytest.mark.parametrize("T,I,O,launches", [
    (1920, 1000, 5456, 1), (700, 2200, 2000, 1), (768, 848, 848, 1), (512, 256, 512, 1), (1, 8, 8, 1), (512, 256, 1024, 1), (768, 256, 248, 1),
    (130, 264, 2048, 1), (257, 136, 1000, 1), (4096, 128, 1024, 1), (1024, 512, 1024, 1), (512, 1024, 1024, 1),
    (4096, 1024, 1024, 2), (2048, 256, 4096, 2), (333, 1024, 3000, 2)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_two_products_same_bits(T, I, O, launches, accumulate):
    import ctypes
    from cai_b200 import ops
    from cai_b200.ops import _lib
    torch.manual_seed(3)
    x, dy, w = (torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((T, I), (T, O), (O, I)))
    dw = torch.randn(O, I, device="cuda")
    res = torch.randn(T, I, device="cuda").to(torch.bfloat16) if accumulate else None
    stream = torch.cuda.current_stream().cuda_stream
    for order in (1, -1):
        calls = [_call(x, w, dy, residual=res), _call(x, w, dy, dw, accumulate)][::order]
        cols = ctypes.c_int()
        a, b = (ctypes.byref(c[0]) for c in calls)
        assert ops.lib().cai_gemm_bf16_two_launches(a, b, ctypes.byref(cols)) == launches, cols.value
        assert ops.lib().cai_gemm_bf16_two(a, b, stream) == 0
        assert ops.device_status() == 0
        for _, out, alone in calls:
            assert torch.equal(out, alone)


# The gate / up projection with SwiGLU in its epilogue at widths that are no multiple of a tile: the bits of the product and the stand-alone
# kernel, and nothing beside the results. One feature group, edges of 64 and 128 features, several waves, one row.
@pytest.mark.parametrize("F", [8, 56, 64, 72, 120, 136, 200, 1000, 2728])
@pytest.mark.parametrize("M,K", [(1, 64), (300, 264), (1920, 1000)])
def test_swiglu_of_any_width(M, K, F):
    import ctypes
    from cai_b200 import ops
    out = [ctypes.c_int() for _ in range(3)]
    ops.lib().cai_gemm_bf16_form(M, 2 * F, K, 1, 0, 0, 148, 0, *map(ctypes.byref, out))
    torch.manual_seed(4)
    x, w = (torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((M, K), (2 * F, K)))
    gu, act = torch.full((M + 1, 2 * F), 5.0, device="cuda").to(torch.bfloat16), torch.full((M + 1, F), 5.0, device="cuda").to(torch.bfloat16)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (x, w, gu, act)]
    q = ctypes.c_longlong
    assert ops.lib().cai_gemm_bf16_swiglu(*p, M, F, K, q(K), q(K), q(2 * F), q(F), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = ops.gemm(x, w)
    if out[1].value == 1:
        assert torch.equal(gu[:M], want)
    assert torch.equal(act[:M], ops.swiglu_fwd(gu[:M].contiguous()))
    assert torch.allclose(gu[:M].float(), want.float(), rtol=2.0 ** -7, atol=1e-2)
    assert bool((gu[M] == 5.0).all()) and bool((act[M] == 5.0).all())
    assert ops.device_status() == 0


# The gate / up projection with SwiGLU over ragged slabs (the C entry): live rows as without slabs, bit for bit, and nothing in halves of tiles past a count.
@pytest.mark.parametrize("slabs,seg_rows,F,K", [(4, 256, 128, 64), (3, 384, 384, 264), (8, 128, 256, 1000)])
@pytest.mark.parametrize("kind", ["none", "full", "edges", "random"])
def test_swiglu_of_ragged_rows(slabs, seg_rows, F, K, kind):
    import ctypes
    from cai_b200 import ops
    g = torch.Generator().manual_seed(slabs + F)
    counts = {"none": torch.zeros(slabs), "full": torch.full((slabs,), seg_rows), "edges": torch.tensor([1, 128, 129, seg_rows - 1, 127, 0, 64, 2])[:slabs],
              "random": torch.randint(0, seg_rows + 1, (slabs,), generator=g)}[kind].to(torch.int32)
    M, c = slabs * seg_rows, counts.cuda()
    x, w = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda(), (torch.randn(2 * F, K, generator=g) * 0.1).to(torch.bfloat16).cuda()
    gu, act = torch.full((M, 2 * F), 5.0, device="cuda", dtype=torch.bfloat16), torch.full((M, F), 5.0, device="cuda", dtype=torch.bfloat16)
    p, q = [ctypes.c_void_p(t.data_ptr()) for t in (x, w, gu, act)], ctypes.c_longlong
    assert ops.lib().cai_gemm_bf16_seg(*p, M, 2 * F, K, q(K), q(K), q(2 * F), q(F), 0, 0, ops.EPI_SWIGLU, ctypes.c_float(1.0), ctypes.c_void_p(c.data_ptr()),
                                       seg_rows, 1, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want_gu, want_act = ops.gemm_swiglu(x, w)
    for s, n in enumerate(counts.tolist()):
        for got, want in ((gu, want_gu), (act, want_act)):
            got, want = got[s * seg_rows:(s + 1) * seg_rows], want[s * seg_rows:(s + 1) * seg_rows]
            assert torch.equal(got[:n], want[:n]) and bool((got[(n + 127) // 128 * 128:] == 5.0).all())
    assert ops.device_status() == 0

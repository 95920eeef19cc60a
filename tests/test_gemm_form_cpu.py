"""The form a bf16 product runs in follows from its shape alone: asked here, where there is no GPU to look at."""
import ctypes
import random

import pytest

from cai_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib._LIB_PATH.exists(), reason="kernel library not built")

EPI_BF16, EPI_SWIGLU, EPI_SWIGLU_BWD = 0, 4, 5


def ask(M, N, K, groups=1, epi=EPI_BF16, segmented=0, sms=148, limit=0):
    out = [ctypes.c_int() for _ in range(3)]
    rc = _lib.lib().cai_gemm_bf16_form(M, N, K, groups, epi, segmented, sms, limit, *map(ctypes.byref, out))
    return tuple(v.value for v in out) if rc == 0 else rc


def form(*args, **kw):
    r = ask(*args, **kw)
    return r if isinstance(r, int) else r[:2]


# tiles of 256 x 128, K -> columns of a tile and slices of K; both sides of each line the rule draws
@pytest.mark.parametrize("M,N,K,want", [
    (256, 256, 256, (128, 1)), (333, 1024, 3000, (128, 2)),           # short K; 16 tiles
    (256, 1920, 2048, (128, 4)), (256, 2048, 2048, (128, 2)),         # 15 and 16 tiles
    (768, 1408, 2048, (128, 2)), (512, 2176, 2048, (128, 1)),         # 33 and 34
    (1536, 1536, 2048, (128, 1)), (1280, 2048, 2048, (256, 1)),       # 72 and 80: one wave of narrow tiles, two
    (8192, 8192, 8192, (256, 1)), (40, 3000, 512, (128, 1)), (1, 8, 8, (128, 1)),
])
def test_form_by_shape(M, N, K, want):
    assert form(M, N, K) == want


def test_split_only_where_sums_are_plain():
    assert form(256, 1920, 2048, epi=EPI_SWIGLU) == (256, 1)
    assert form(256, 1920, 2048, segmented=1)[1] == 1
    assert form(256, 128, 2048, groups=40)[1] == 1 and form(256, 128, 2048, groups=15)[1] == 4
    assert form(256, 128, 128, epi=EPI_SWIGLU_BWD) < 0 and form(0, 128, 128) < 0


# (M, N, K): persistent wide, persistent narrow, two and four slices
@pytest.mark.parametrize("shape,cluster,free", [((8192, 8192, 8192), 2, 148), ((1536, 1536, 2048), 2, 144), ((333, 1024, 3000), 4, 64),
                                                ((768, 1408, 2048), 4, 132), ((256, 1920, 2048), 8, 120)])
def test_limit_caps_the_ctas(shape, cluster, free):
    assert ask(*shape)[2] == free
    for limit in (1, 2, 3, 7, 8, 15, 16, 33, 100, 131, 147, 148, 1000):
        f = ask(*shape, limit=limit)
        assert f[:2] == ask(*shape)[:2] == ask(*shape, sms=132)[:2]        # the sums do not depend on the limit or the GPU
        most = max(cluster, min(limit, 148) // cluster * cluster)         # whole clusters; one at least
        assert f[2] == min(free, most), (limit, f)


def walk(M, N, groups, counts, seg_rows, tile_cols, pairs):
    """Every pair's tiles: (group, column tile, row of each half, whether it is live)."""
    c = (ctypes.c_int * len(counts))(*counts)
    out, per_pair = [], []
    for pair in range(pairs):
        ask_walk = lambda buf, n: _lib.lib().cai_gemm_bf16_ragged_walk(M, N, groups, c, seg_rows, tile_cols, pairs, pair, buf, n)
        n = ask_walk(None, 0)
        assert n >= 0
        buf = (ctypes.c_int * max(1, 6 * n))()
        assert ask_walk(buf, n) == n
        out += [tuple(buf[6 * i:6 * i + 6]) for i in range(n)]
        per_pair.append(n)
    return out, per_pair


# (groups, slabs per group, rows of a slab, rows of the group if less): live halves counted ahead, up to 256 slabs, and the walk over all
# tiles beyond. Slabs of odd numbers of halves, one slab and several, more row tiles than a raster group, a last slab cut short.
@pytest.mark.parametrize("groups,per,seg_rows,short", [(1, 1, 128, 0), (8, 8, 128, 0), (5, 3, 384, 0), (4, 4, 256, 100), (2, 2, 2432, 0), (1, 256, 128, 0),
                                                       (64, 1, 2048, 0), (256, 1, 128, 60), (300, 1, 128, 0), (2, 130, 384, 0)])
@pytest.mark.parametrize("kind", ["full", "none", "one", "random", "edges"])
def test_ragged_walk_covers_live_halves_once(groups, per, seg_rows, short, kind):
    rng = random.Random(groups * 31 + per)
    n = groups * per
    edges = [0, 1, 127, 128, 129, 255, 256, 257, seg_rows - 1, seg_rows, seg_rows + 5, -1]
    counts = {"full": [seg_rows] * n, "none": [0] * n, "one": [seg_rows if i == n // 2 else 0 for i in range(n)],
              "random": [rng.randint(0, seg_rows) for _ in range(n)], "edges": [edges[i % len(edges)] for i in range(n)]}[kind]
    M, N, tile_cols, pairs = per * seg_rows - short, 640, 256, 74
    tiles, per_pair = walk(M, N, groups, counts, seg_rows, tile_cols, pairs)
    want = set()
    for i, c in enumerate(counts):
        first = i % per * seg_rows
        want |= {(i // per, tn, first + r) for r in range(0, min(c, seg_rows, M - first), 128) for tn in range(3)}
    got = [(g, tn, row) for g, tn, r0, r1, l0, l1 in tiles for row, live in ((r0, l0), (r1, l1)) if live]
    assert len(got) == len(set(got)) and set(got) == want
    assert all(0 <= r < M and r % 128 == 0 for t in tiles for r in t[2:4] if n <= 256)       # a half that is not live is loaded all the same
    if n <= 256:
        halves = [len({h for h in want if h[0] == g and h[1] == 0}) for g in range(groups)]
        assert len(tiles) == 3 * sum((h + 1) // 2 for h in halves)            # no half-empty tile but the last of a group
        assert max(per_pair) - min(per_pair) <= 1


def two_walk(n0, k0, n1, k1, cols, pairs):
    per_pair = []
    for pair in range(pairs):
        ask_walk = lambda buf, n: _lib.lib().cai_gemm_bf16_two_walk(n0, k0, n1, k1, cols, pairs, pair, buf, n)
        n = ask_walk(None, 0)
        buf = (ctypes.c_int * (2 * max(n, 1)))()
        assert ask_walk(buf, n) == n
        per_pair.append([(buf[2 * i], buf[2 * i + 1]) for i in range(n)])
    return per_pair


# Two products in one launch: every tile once, the longer tiles of a pair first, and no pair done later than a list ordered by length allows
# (the average and one tile of either kind). Tile counts around whole rounds of the pairs, none of the second, one of each, K from equal to 64 times.
@pytest.mark.parametrize("pairs", [1, 2, 74])
@pytest.mark.parametrize("k0,k1", [(512, 512), (4096, 512), (1000, 136), (8192, 128)])
def test_two_products_walk(pairs, k0, k1):
    for n0 in (1, 2, 32, 73, 74, 75, 148, 149, 500):
        for n1 in (0, 1, 5, 73, 74, 88, 147, 1000):
            if n0 + n1 < pairs:
                continue
            walks = two_walk(n0, k0, n1, k1, 256, pairs)
            assert sorted(t for w in walks for t in w) == [(0, i) for i in range(n0)] + [(1, i) for i in range(n1)]
            c = [(k + 127) // 128 * 1150.0 + 2500.0 for k in (k0, k1)]
            load = [sum(c[which] for which, _ in w) for w in walks]
            assert all(w == sorted(w) for w in walks)
            assert max(load) <= (n0 * c[0] + n1 * c[1]) / pairs + c[0] + c[1]


def gemm_call(M, N, K, epi=EPI_BF16):
    return _lib.GemmCall(M=M, N=N, K=K, epi=epi, alpha=1.0)


def two_launches(a, b):
    cols = ctypes.c_int()
    return _lib.lib().cai_gemm_bf16_two_launches(ctypes.byref(a), ctypes.byref(b), ctypes.byref(cols)), cols.value


def test_two_products_launches():
    assert two_launches(gemm_call(1920, 1000, 5456), gemm_call(5456, 1000, 1920)) == (1, 256)     # 32 and 88 tiles: waves fill up
    assert two_launches(gemm_call(4096, 2048, 8192), gemm_call(8192, 2048, 4096))[0] == 2         # at the power limit
    assert two_launches(gemm_call(3456, 1408, 2944), gemm_call(2944, 1408, 3456))[0] == 2         # as many waves as apart
    assert two_launches(gemm_call(768, 848, 848), gemm_call(848, 848, 768)) == (1, 128)           # one wave of narrow tiles
    assert two_launches(gemm_call(512, 256, 1024), gemm_call(1024, 256, 512)) == (1, 128)         # 4 clusters of four slices, 8 tiles of one sum
    assert two_launches(gemm_call(256, 1920, 2048), gemm_call(768, 1408, 2048))[0] == 2           # 15 clusters of four slices, 33 tiles of two
    assert two_launches(gemm_call(256, 1792, 2048), gemm_call(256, 512, 512)) == (1, 128)         # 14 and one more with four tiles of one sum
    assert two_launches(gemm_call(256, 1792, 2048), gemm_call(256, 640, 512))[0] == 2
    assert two_launches(gemm_call(512, 512, 512), gemm_call(512, 512, 512, EPI_SWIGLU))[0] == 2
    assert two_launches(gemm_call(0, 512, 512), gemm_call(512, 512, 512))[0] == 1

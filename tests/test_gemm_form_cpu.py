"""The form a bf16 product runs in follows from its shape alone: asked here, where there is no GPU to look at."""
import ctypes

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

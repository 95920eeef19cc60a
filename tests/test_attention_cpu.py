"""The form the attention forward runs in follows from its grid: asked here, where there is no GPU to look at."""
import pytest

from cai_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib._LIB_PATH.exists(), reason="kernel library not built")


# Rows between one wave of one-tile CTAs and one of two-tile CTAs on 148 SMs, measured in every form: the fastest of each (both where they
# are within 2 %), on both sides of the line for each length
@pytest.mark.parametrize("S,heads,best", [
    (256, 83, {2, 3}), (256, 145, {2}), (384, 50, {2, 3}), (384, 70, {2}),
    (512, 38, {1, 3}), (512, 45, {3}), (512, 73, {3}),
    (640, 30, {1}), (640, 33, {1}), (640, 39, {3}), (640, 46, {2, 3}),
    (768, 30, {1}), (768, 35, {1, 3}), (768, 39, {3}),
    (896, 26, {1}), (896, 30, {1, 3}), (896, 33, {3}),
    (1024, 19, {1}), (1024, 27, {1}), (1024, 32, {3}),
    (1152, 24, {1}), (1152, 28, {1, 3}), (1280, 23, {1}), (1280, 25, {1, 3}), (1280, 29, {3}),
    (1536, 13, {1}), (1536, 21, {1}), (1536, 23, {1, 3}), (1792, 11, {1}), (1792, 20, {1}), (1920, 10, {1}), (1920, 18, {1})])
def test_form_of_grids_that_overflow_a_wave(S, heads, best):
    assert 148 < S // 128 * heads < 296
    for B in (1, heads):
        assert _lib.lib().cai_flash_attn_fwd_form(B, S, heads // B, 148) in best


def test_form_of_small_and_large_grids():
    form = _lib.lib().cai_flash_attn_fwd_form
    assert form(1, 128, 1, 148) == form(4, 128, 36, 148) == form(1, 2048, 9, 148) == form(1, 8192, 2, 148) == 1
    assert form(1, 128, 148, 148) == form(1, 2048, 32, 148) == form(4, 4096, 16, 148) == 3
    assert form(1, 8192, 32, 148) == 2

"""The package's front door: public names resolve lazily, and importing the package needs no GPU and no torch."""
import subprocess
import sys
import sysconfig
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_import_is_light_and_public_names_resolve():
    code = ("import sys, cai_b200\n"
            "assert 'torch' not in sys.modules, 'importing the package must not pull torch in'\n"
            "for n in cai_b200.__all__: assert getattr(cai_b200, n) is not None, n\n"
            "assert cai_b200.plan.PlanFile is cai_b200.PlanFile\n"
            "print(cai_b200.__version__)\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip()


def test_ops_import_with_a_torch_that_has_no_cuda():
    """The two stream functions of a CUDA build are looked up when an op is called."""
    code = ("import torch\n"
            "for n in ('_cuda_getDevice', '_cuda_getCurrentRawStream'):\n"
            "    if hasattr(torch._C, n): delattr(torch._C, n)\n"
            "import cai_b200.ops\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_unknown_attribute_is_an_attribute_error():
    import cai_b200
    with pytest.raises(AttributeError):
        cai_b200.no_such_thing
    assert not hasattr(cai_b200, "__wrapped__")


def test_log_level_from_the_environment_and_the_api(tmp_path):
    """CAI_LOG_LEVEL sets the native library's starting level; set_log_level overrides it."""
    import os
    code = ("from cai_b200 import plan\n"
            "import sys\n"
            "if len(sys.argv) > 1: plan.set_log_level(sys.argv[1])\n"
            f"plan.compile_plans(open('{ROOT}/configs/tiny.cfg').read(), '{tmp_path}', ranks=(0, 1), version=2, text=True)\n"
            f"s = plan.Simulator('{tmp_path}/plan.rank000000.bin', '{tmp_path}/topology.bin', rank=0)\n"
            "s.step(); s.close()\n")
    def run(env_level=None, arg=None):
        env = {k: v for k, v in os.environ.items() if k != "CAI_LOG_LEVEL"}
        if env_level:
            env["CAI_LOG_LEVEL"] = env_level
        r = subprocess.run([sys.executable, "-c", code] + ([arg] if arg else []), capture_output=True, text=True, cwd=ROOT, env=env, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stderr
    assert "[cai INFO] plan loaded" in run()
    assert "[cai INFO]" not in run(env_level="warn")
    assert "[cai INFO]" not in run(env_level="0")
    assert "[cai INFO] plan loaded" in run(env_level="warn", arg="info")
    assert "[cai INFO]" not in run(arg="error")


def test_launchers_of_the_extension_are_those_of_the_library():
    """The extension the ops call through against ctypes: same results and errors for calls that need no GPU, arguments taken alike."""
    from cai_b200.ops import _lib
    if not _lib._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    fast, slow = _lib.calls(), _lib.lib()
    if not (Path(sysconfig.get_paths()["include"]) / "Python.h").exists():
        pytest.skip("no Python header to build the extension with")
    assert fast is not slow
    for rows in (1, 100, 5000, True):
        assert fast.cai_rmsnorm_bwd_parts(rows) == slow.cai_rmsnorm_bwd_parts(rows)
    bad = (None, 0, 16, None, 16, 12, 16, 16, 16, 16, 0, 0, False, 0, 1, 0, None)     # N not a multiple of 8; null pointers, an integer for a float
    assert fast.cai_gemm_bf16(*bad) == slow.cai_gemm_bf16(*bad) < 0
    assert b"multiples of 8" in slow.cai_last_error()
    empty = (0, 0, 0, 0, -1, 16, 16, 1 << 40, 16, 16, 0, 0, 0, 0, 1.0, 0, 0)          # nothing to do
    assert fast.cai_gemm_bf16(*empty) == slow.cai_gemm_bf16(*empty) == 0
    with pytest.raises(TypeError):
        fast.cai_gemm_bf16(*bad[:-1])
    with pytest.raises(TypeError):
        fast.cai_gemm_bf16("x", *bad[1:])
    with pytest.raises(TypeError):
        fast.cai_gemm_bf16(*bad[:4], 1.5, *bad[5:])


def test_an_extension_that_cannot_be_loaded_is_an_error(tmp_path, monkeypatch):
    """Not a silent way to ctypes, which is for where none was built."""
    from cai_b200.ops import _lib
    if not _lib._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    slow = _lib.lib()
    monkeypatch.setattr(_lib, "_LIB_PATH", tmp_path / "libcai_kernels.so")
    monkeypatch.setattr(_lib, "_calls", None)
    assert _lib.calls() is slow
    (tmp_path / ("_calls" + sysconfig.get_config_var("EXT_SUFFIX"))).write_bytes(b"no shared object")
    for _ in range(2):
        monkeypatch.setattr(_lib, "_calls", None)
        with pytest.raises(ImportError):
            _lib.calls()


# RMSNorm backward whose rows come ahead: which rows a CTA fetches and works on. Row groups of 8, 4 and 1, CTAs without rows, a last round that is not full.
@pytest.mark.parametrize("rows,H,ctas", [(4737, 8, 296), (100, 1000, 3), (2500, 1032, 7), (650, 8192, 296), (5, 1000, 2)])
def test_norm_rows_that_do_not_come_end_the_ctas_work(rows, H, ctas):
    import ctypes
    from cai_b200.ops import _lib
    if not _lib._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    groups = 8 if H <= 1024 else 4 if H <= 2048 else 1

    def events(cta, lost):
        n = _lib.lib().cai_rmsnorm_bwd_rounds(rows, H, ctas, cta, lost, None, 0)
        buf = (ctypes.c_int * (2 * max(n, 1)))()
        assert _lib.lib().cai_rmsnorm_bwd_rounds(rows, H, ctas, cta, lost, buf, n) == n
        return [(buf[2 * i], buf[2 * i + 1]) for i in range(n)]

    worked = []
    for cta in range(ctas):
        whole = events(cta, -1)
        mine = list(range(cta * groups, rows, ctas * groups))
        assert [r for what, r in whole if what == 0] == mine and [r for what, r in whole if what == 1] == mine
        worked += mine
        for lost in range(len(mine)):
            # this round's rows were fetched; nothing is done with them, and nothing is fetched over them
            want = [(0, mine[0])] + [e for k in range(lost) for e in ((0, mine[k + 1]), (1, mine[k]))]
            assert events(cta, lost) == want
    assert sorted(worked) == list(range(0, rows, groups))


# Rows of the vocabulary a CTA of the embedding backward takes: the faster of the two where they were measured apart, on both sides of each line the rule draws
@pytest.mark.parametrize("T,rows,H,best", [
    (512, 512, 256, 8), (256, 1184, 128, 8), (256, 3000, 128, 32), (512, 9472, 256, 32), (1024, 5000, 128, 32), (3000, 2368, 128, 8), (8192, 7000, 256, 32),
    (256, 2368, 384, 8), (256, 4736, 264, 32), (1024, 4736, 512, 32), (8192, 4736, 512, 8), (16384, 7000, 512, 32),
    (256, 3000, 640, 8), (256, 4736, 768, 32), (3000, 6000, 768, 8), (8192, 9472, 768, 32),
    (3840, 5000, 1000, 8), (64, 9472, 1400, 8), (16384, 9472, 4096, 8), (4096, 32000, 1024, 32), (512, 16000, 256, 32)])
def test_rows_of_an_embedding_cta(T, rows, H, best):
    from cai_b200.ops import _lib
    if not _lib._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    assert _lib.lib().cai_embed_bwd_rows(T, rows, H, 1, 148) == best


@pytest.mark.parametrize("T,pieces,rows_an_sm", [(1, 1, 8), (1023, 1, 8), (1024, 1, 12), (2047, 1, 12), (2048, 1, 16), (1023, 2, 16), (2048, 2, 32), (2048, 3, 48), (1, 4, 64)])
def test_lines_of_the_embedding_rule(T, pieces, rows_an_sm):
    from cai_b200.ops import _lib
    if not _lib._LIB_PATH.exists():
        pytest.skip("kernel library not built")
    rows = _lib.lib().cai_embed_bwd_rows
    for H, wide in ((256 * pieces, 1), (256 * pieces - 248, 1), (32 * pieces, 0), (32 * pieces - 31, 0)):
        assert rows(T, rows_an_sm * 148, H, wide, 148) == 8 and rows(T, rows_an_sm * 148 + 1, H, wide, 148) == 32

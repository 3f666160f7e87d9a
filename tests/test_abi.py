"""The C-ABI library builds, loads without a GPU and exports every symbol include/stu_b200.h declares."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "stu_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(?:int|long long)\s+(stu_\w+)\s*\(", text)))


def test_header_declares_entry_points():
    names = declared_symbols()
    assert "stu_linear" in names and "stu_decode_approx" in names and len(names) >= 10


def test_library_exports_every_declared_symbol():
    from flash_stu_2_b200 import _lib
    lib = _lib.load()
    raw = ctypes.CDLL(_lib.LIB_PATH)
    for name in declared_symbols():
        assert hasattr(raw, name), f"{name} declared in include/stu_b200.h but not exported"
    # the Python binding covers exactly the declared set
    assert sorted(_lib.exported_symbols()) == declared_symbols()
    assert lib.stu_b200_version() >= 100


def test_argument_errors_are_reported_without_a_gpu():
    from flash_stu_2_b200 import _lib
    lib = _lib.load()
    # null pointers / bad shapes are rejected on the host before any CUDA call
    assert lib.stu_rmsnorm(None, None, None, 1, 8, 8, 8, 1e-6, 1, None) == -5
    assert lib.stu_linear_can_fuse_norm(8, 4096, 1024, 2, 1) == 1
    assert lib.stu_linear_can_fuse_norm(8, 4096, 1024, 2, 0) == 0
    assert lib.stu_linear_can_fuse_norm(128, 4096, 1024, 2, 1) == 0
    # the prefill convolution reads its scratch in 16-byte vectors: a row pitch that is not a multiple of 8 bf16
    # (4 fp32) elements, or a misaligned scratch base, is refused with -3 and nothing is launched
    a = 0x10000   # stands for an aligned device address; the checks return before anything dereferences it
    assert lib.stu_conv_prefill_approx(a, a, a, a, 333 * 8, 8, 1, 8, 168, 167, 0, 333, 1, 1, None) == -3
    assert lib.stu_conv_prefill_approx(a, a, a, a, 333 * 8, 8, 1, 8, 168, 166, 0, 332, 0, 0, None) == -3
    assert lib.stu_conv_prefill_approx(a, a, a + 2, a, 333 * 8, 8, 1, 8, 168, 168, 0, 333, 1, 1, None) == -3
    # the tcgen05 convolution: misaligned scratch -3, a history that is not tiled in 128-position blocks -4, fp32 -1
    assert lib.stu_conv_prefill_approx_tc5(a, a, a + 2, a, 333 * 8, 8, 1, 8, 256, 168, 0, 333, None, 1, None) == -3
    assert lib.stu_conv_prefill_approx_tc5(a, a, a, a, 333 * 8, 8, 1, 8, 168, 168, 0, 333, None, 1, None) == -4
    assert lib.stu_conv_prefill_approx_tc5(a, a, a, a, 333 * 8, 8, 1, 8, 256, 168, 0, 333, None, 0, None) == -1


def test_programmatic_launch_switch_round_trips_without_a_gpu():
    """stu_set_programmatic_launch returns the previous setting; the token-step kernels read it at launch time."""
    from flash_stu_2_b200 import ops
    prev = ops.set_programmatic_launch(False)
    try:
        assert ops.set_programmatic_launch(True) is False
        assert ops.set_programmatic_launch(True) is True
    finally:
        ops.set_programmatic_launch(prev)


def test_linear_bench_module_imports_without_a_gpu():
    import torch
    import flash_stu_2_b200.linear_bench as lb
    if torch.cuda.is_available():
        pytest.skip("with a GPU the module would run its measurement")
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        lb.main([])


def test_ops_refuse_cpu_tensors():
    import torch
    from flash_stu_2_b200 import ops
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops.rmsnorm(torch.randn(2, 8), torch.ones(8))


def test_extension_module_calls_the_same_functions():
    """The entry points of the extension module return what ctypes gets, take None, addresses and keyword-free integers and
    floats, and refuse a wrong number of arguments, values that do not convert and tensors that are not on a GPU."""
    import torch
    from flash_stu_2_b200 import _lib, ops
    lib, native = _lib.load(), _lib.native()
    assert native.stu_rmsnorm(None, None, None, 1, 8, 8, 8, 1e-6, 1, None) == lib.stu_rmsnorm(None, None, None, 1, 8, 8, 8, 1e-6, 1, None) == -5
    assert native.stu_linear_can_fuse_norm(8, 4096, 1024, 2, True) == 1
    a = 0x10000
    args = (a, a, a + 2, a, 333 * 8, 8, 1, 8, 256, 168, 0, 333, None, 1, None)
    assert native.stu_conv_prefill_approx_tc5(*args) == lib.stu_conv_prefill_approx_tc5(*args) == -3
    with pytest.raises(TypeError, match="arguments expected"):
        native.stu_linear_can_fuse_norm(8, 4096)
    with pytest.raises(TypeError):
        native.stu_linear_can_fuse_norm(8, 4096, 1024, 2, "bf16")
    with pytest.raises(OverflowError):
        native.stu_linear_can_fuse_norm(8, 1 << 40, 1024, 2, 1)
    x = torch.zeros(2, 8)
    with pytest.raises(RuntimeError, match="no CPU path"):
        native.stu_rmsnorm(x, x, x, 2, 8, 8, 8, 1e-6, 0, None)
    assert native.linear(x, x, None, None, None, 0, None, 1e-6, 0, False, 0, 0, 0) is None and native.rmsnorm(x, x, 1e-6) is None
    for call in (lambda: ops.linear(x, x), lambda: ops.rmsnorm(x, x[0])):
        with pytest.raises(RuntimeError, match="no CPU path"):
            call()
    exported = set(dir(native))
    used = set(re.findall(r"_lib\.native\(\)\.(\w+)\(", open(os.path.join(ROOT, "flash_stu_2_b200", "ops.py")).read()))
    assert used <= exported, used - exported


def test_long_inputs_of_the_fp32_convolutions_are_not_refused():
    """More tiles of positions than a grid's second dimension holds.  (The addresses are dummies: only where no launch can reach them.)"""
    import torch
    from flash_stu_2_b200 import _lib
    if torch.cuda.is_available():
        pytest.skip("would be launched")
    call = lambda t_end: _lib.load().stu_full_conv(0x10000, t_end // 2 + 4 & ~3, 0x10000, 64, 2, 0x10000, 16, 1, 8, 0, 0, t_end, 0, None)
    assert call(1000) > 0 and call(9_000_000) == call(1000)   # CUDA's own error: no device


def test_a_missing_extension_module_is_reported_like_a_missing_library(monkeypatch):
    import sys
    import flash_stu_2_b200
    from flash_stu_2_b200 import _lib
    _lib.native()
    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.delattr(flash_stu_2_b200, "_native", raising=False)
    monkeypatch.setitem(sys.modules, "flash_stu_2_b200._native", None)   # its import fails
    with pytest.raises(RuntimeError, match="no CPU fallback; run"):
        _lib.native()


def test_the_extension_module_is_stale_for_another_torch(monkeypatch):
    """A torch installed after the module was built: it is built again."""
    from flash_stu_2_b200 import _build, _lib
    _lib.native()
    assert not _build.native_stale()
    import torch
    real = os.path.getmtime
    version = os.path.join(os.path.dirname(torch.__file__), "version.py")
    assert os.path.exists(version)
    monkeypatch.setattr(_build.os.path, "getmtime", lambda p: real(p) + (1e9 if os.path.samefile(p, version) else 0))
    assert _build.native_stale()

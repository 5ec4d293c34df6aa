"""The native operator calls of the Python binding against the ctypes ones: the same refusals, the same reading of integers, and
arguments that only ctypes can judge left to it. No GPU: every call ends at the null runtime handle."""
import ctypes as C

import numpy as np
import pytest

from tessl_b200 import capi, nn

try:
    capi.load()
except ImportError:
    pytest.skip("the library is not built", allow_module_level=True)


class NullRuntime:
    handle = None


B = nn.GpuBuffer(4096, 1 << 20)
BANK = nn.Q4MlxBank(B, B)
SHAPE = nn.QuantShape(8, 64, 32)
OUT = nn.QkvOutputs(B, B, B)
CALLS = {
    "gemv_q4_mlx_simd": (nn.gemv_q4_mlx_simd, (BANK, B, B, SHAPE)),
    "gemv_q4_mlx_gate_up_silu": (nn.gemv_q4_mlx_gate_up_silu, (BANK, BANK, B, B, SHAPE, True)),
    "gemv_q4_mlx_kv": (nn.gemv_q4_mlx_kv, (BANK, BANK, B, B, B, SHAPE)),
    "gemv_q4_mlx_qkv": (nn.gemv_q4_mlx_qkv, (BANK, BANK, BANK, B, OUT, 8, 8, 64, 32)),
    "swiglu": (nn.swiglu, (B, B, B, 8, False)),
    "gemm_q4_mlx": (nn.gemm_q4_mlx, (BANK, B, B, SHAPE, 2)),
    "gemm_q4_mlx_tensorops": (nn.gemm_q4_mlx_tensorops, (BANK, B, B, SHAPE, 9)),
    "gemv_q8": (nn.gemv_q8, (B, B, B, B, B, 8, 64, 32)),
    "gemm_q8_mlx": (nn.gemm_q8_mlx, (B, B, B, B, SHAPE, 2)),
    "embed_lookup_q4_mlx": (nn.embed_lookup_q4_mlx, (BANK, B, B, 8, 64, 32, 1)),
    "qwen35_rms_norm": (nn.qwen35_rms_norm, (B, B, B, True, 1, 64, 1e-6)),
    "qwen35_residual_add": (nn.qwen35_residual_add, (B, B, 1, 64)),
    "qwen35_add_rms_norm": (nn.qwen35_add_rms_norm, (B, B, B, B, True, 1, 64, 1e-6)),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_each_call_reaches_the_library(name, monkeypatch):
    fn, args = CALLS[name]
    monkeypatch.setattr(capi, "call", lambda *a: pytest.fail("went through ctypes"))
    for rt in (NullRuntime(), type("R", (), {"handle": C.c_void_p(None)})()):
        with pytest.raises(nn.TesslError, match="null runtime handle") as e:
            fn(rt, *args)
        assert e.value.status == capi.TESSL_ERR and isinstance(e.value, RuntimeError)


@pytest.mark.parametrize("name", sorted(CALLS))
def test_what_it_cannot_read_goes_through_ctypes(name):
    """A first argument, or a runtime, that is none: the same exception as before."""
    fn, args = CALLS[name]
    with pytest.raises(AttributeError):
        fn(NullRuntime(), object(), *args[1:])
    with pytest.raises(AttributeError):
        fn(object(), *args)


def test_flags_and_numbers_of_other_types_are_left_to_ctypes():
    native, rt = capi.native(), NullRuntime()
    assert native.swiglu(rt, B, B, B, np.int64(8), False) is False
    assert native.swiglu(rt, B, B, B, 8, 1) is False
    assert native.swiglu(rt, B, B, B, 8.0, False) is False
    assert native.qwen35_rms_norm(rt, B, B, B, True, 1, 64, 1) is False
    assert native.swiglu(rt, B, B, B, 8) is False
    bad = nn.GpuBuffer(4096, 16)
    bad.nbytes = "many"
    assert native.swiglu(rt, bad, B, B, 8, False) is False


def test_integers_wrap_as_ctypes_arguments_do():
    for n in (-1, 2**32, 2**40 + 3):
        with pytest.raises(nn.TesslError, match="null runtime handle"):
            nn.swiglu(NullRuntime(), B, B, B, n, False)


def test_the_module_has_what_the_binding_calls():
    native = capi.native()
    assert native.ABI_VERSION == capi.ABI_VERSION
    assert sorted(capi.NATIVE_OPERATORS) == sorted(CALLS) and all(callable(getattr(native, n)) for n in CALLS)


@pytest.mark.parametrize("name", sorted(CALLS))
def test_without_the_module_every_call_goes_through_ctypes(name, monkeypatch, tmp_path):
    """A module that was not built, or only for another interpreter, whose file has another name."""
    import shutil

    shutil.copy(capi.CALL_PATH, tmp_path / "_tessl_call.cpython-27-elsewhere.so")
    monkeypatch.setattr(capi, "CALL_PATH", tmp_path / capi.CALL_PATH.name)
    monkeypatch.setattr(nn, "_native", nn._Native())
    fn, args = CALLS[name]
    with pytest.warns(RuntimeWarning, match="through ctypes"), pytest.raises(nn.TesslError, match="null runtime handle"):
        fn(NullRuntime(), *args)
    with pytest.raises(AttributeError):
        fn(object(), *args)


def test_a_module_of_another_abi_is_not_used(monkeypatch):
    monkeypatch.setattr(capi, "ABI_VERSION", capi.ABI_VERSION + 1)
    with pytest.warns(RuntimeWarning, match="has ABI"):
        assert capi.native() is None


def test_the_build_goes_on_without_the_module(monkeypatch, tmp_path, capsys):
    from tessl_b200 import build

    monkeypatch.setattr(build, "is_stale", lambda: False)
    monkeypatch.setattr(build, "PY_CALL", tmp_path / "absent")
    monkeypatch.setattr(build, "build_py_call", lambda: (_ for _ in ()).throw(RuntimeError("no C compiler found")))
    assert build.build() == build.LIB
    assert "ctypes: no C compiler found" in capsys.readouterr().err


def test_another_interpreter_builds_its_own_module():
    import sysconfig

    from tessl_b200 import build

    assert build.PY_CALL == capi.CALL_PATH and build.PY_CALL.name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))

"""The CPython face of the hot entry points: the same functions as through ctypes, and its argument checks."""

import sys
import sysconfig
from pathlib import Path

import pytest

import mlx_batch_invariant_b200
from mlx_batch_invariant_b200 import _lib, build


def test_the_same_answers_as_through_ctypes():
    c, l = _lib.calls(), _lib.load()
    for M, N, K in ((1, 4096, 4096), (64, 4096, 14336), (300, 4096, 4096), (100, 4096, 4096)):
        for dt in (_lib.BI_F32, _lib.BI_F16, _lib.BI_BF16):
            assert c.bi_matmul_scratch_bytes(M, N, K, dt) == l.bi_matmul_scratch_bytes(M, N, K, dt)
            assert c.bi_qmm_scratch_bytes(M, N, K, dt) == l.bi_qmm_scratch_bytes(M, N, K, dt)
    assert c.bi_attn_decode_workspace_bytes(2, 32, 257, 128, 256) == l.bi_attn_decode_workspace_bytes(2, 32, 257, 128, 256)


ENTRIES = ["bi_rms_norm", "bi_add_rms_norm", "bi_matmul", "bi_matmul_bias", "bi_qmm", "bi_attn_decode", "bi_attn_prefill"]
SIZES = ["bi_matmul_scratch_bytes", "bi_qmm_scratch_bytes", "bi_attn_decode_workspace_bytes"]


@pytest.mark.parametrize("name", ENTRIES)
def test_arguments(name):
    """Null pointers (None) are the library's own error, with its message, never a launch; a call takes as many arguments as
    the prototype has, and of their kinds."""
    fn, args = getattr(_lib.calls(), name), _lib.SIGNATURES[name][1]
    values = [0.5 if a is _lib.c_float else None if a is _lib.c_void_p else 1 for a in args]
    code, said = fn(*values), _lib.last_error()
    assert code == getattr(_lib.load(), name)(*values) != _lib.BI_OK
    assert said == _lib.last_error()
    with pytest.raises(TypeError):
        fn(*values[:-1])
    with pytest.raises(TypeError):
        fn(*[0.5] * len(values))
    with pytest.raises(OverflowError):
        fn(*[2 ** 70] * len(values))


@pytest.mark.parametrize("name", ENTRIES + SIZES)
def test_none_is_a_null_pointer_and_nothing_else(name):
    """Slot by slot: None and integers where the prototype has a pointer, numbers where it has one, as through ctypes.
    Integers are zero, so that a call which takes all its arguments does nothing or reports an error."""
    fn, args = getattr(_lib.calls(), name), _lib.SIGNATURES[name][1]
    zeros = [None if a is _lib.c_void_p else 0 for a in args]
    for i, a in enumerate(args):
        for value, pointer, number in ((None, True, False), (0.0, False, a is _lib.c_float), ("0", False, False)):
            values = zeros[:i] + [value] + zeros[i + 1:]
            if pointer if a is _lib.c_void_p else number:
                assert isinstance(fn(*values), int), (i, value)
            else:
                with pytest.raises(TypeError):
                    fn(*values)


def test_the_module_is_this_interpreters():
    """Its name carries the interpreter's ABI tag, so that another Python does not import it."""
    module = Path(_lib.calls().__file__)
    assert module.name == "_calls" + sysconfig.get_config_var("EXT_SUFFIX") and not (module.parent / "_calls.so").exists()


def test_the_library_runs_without_the_module(monkeypatch):
    """A tree with only the library: the same entry points through ctypes, and a warning that says why."""
    monkeypatch.setattr(_lib, "_bound", None)
    monkeypatch.delattr(mlx_batch_invariant_b200, "_calls", raising=False)
    monkeypatch.setitem(sys.modules, "mlx_batch_invariant_b200._calls", None)
    with pytest.warns(RuntimeWarning, match="_calls"):
        c = _lib.calls()
    assert c is _lib.calls() is _lib.load()
    for name in ENTRIES + SIZES:
        assert getattr(c, name).argtypes == _lib.SIGNATURES[name][1]


def test_a_build_without_pythons_headers_has_no_module(monkeypatch, tmp_path, capsys):
    monkeypatch.setattr(build, "CALLS", tmp_path / build.CALLS.name)
    monkeypatch.setattr(build, "OBJ", tmp_path)
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    assert not build.build_calls().exists() and "Python.h" in capsys.readouterr().err

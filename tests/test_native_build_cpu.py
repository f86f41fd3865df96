"""The native host path (heddle_b200._native) saves host time only: what works without it, and when it is built and loaded."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def _python(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return r.stderr


def test_library_loads_without_the_native_module(built_lib):
    err = _python("import sys; sys.modules['heddle_b200._native'] = None\n"
                  "from heddle_b200 import _lib\n"
                  "assert _lib.load().hb_version() == 100 and _lib.native is None")
    assert "host path" in err


def test_native_module_loads_in_front_of_torch(built_lib):
    _python("from heddle_b200 import _lib; _lib.load(); assert _lib.native is not None")


def test_build_goes_on_without_a_compiler(monkeypatch, tmp_path):
    from heddle_b200 import _build

    left = tmp_path / "native.so"
    left.write_text("built from other sources")
    monkeypatch.setattr(_build, "native_path", lambda: left)

    def no_compiler():
        raise FileNotFoundError("g++")

    monkeypatch.setattr(_build, "_compile_native", no_compiler)
    with pytest.warns(RuntimeWarning, match="stays in Python"):
        _build._build_native()
    assert not left.exists() and _build._native_stale()


def test_module_of_another_pytorch_is_neither_fresh_nor_loaded(built_lib, monkeypatch):
    import torch

    from heddle_b200 import _build

    assert not _build._native_stale()
    monkeypatch.setattr(torch, "__version__", "2.99.0")
    assert _build._native_stale()
    err = _python("import torch; torch.__version__ = '2.99.0'\n"
                  "from heddle_b200 import _lib\n"
                  "assert _lib.load().hb_version() == 100 and _lib.native is None")
    assert "host path" in err


def test_module_of_another_python_is_neither_fresh_nor_loaded(built_lib, monkeypatch):
    import sysconfig

    from heddle_b200 import _build

    here = _build.native_path()
    monkeypatch.setitem(sysconfig.get_config_vars(), "EXT_SUFFIX", ".cpython-399-x86_64-linux-gnu.so")
    assert _build.native_path() != here and _build._native_stale()


def test_library_is_built_without_pytorch(built_lib, monkeypatch):
    from heddle_b200 import _build

    def no_torch():
        raise ImportError("No module named 'torch'")

    monkeypatch.setattr(_build, "native_path", no_torch)
    with pytest.warns(RuntimeWarning, match="stays in Python"):
        assert _build.build() == _build.LIB_PATH

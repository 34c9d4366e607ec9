"""The extension module in front of mmv, linear and draft_logits is no condition of the library: where it cannot be had, the Python functions
take every call."""
import os
import subprocess
import sys
import warnings

import pytest

from orin_qwen_lossless_b200 import _lib, build, ops

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_module_is_named_by_what_it_is_bound_to(monkeypatch):
    import torch
    assert torch.__version__ in build.calls_path() and "cpython" in build.calls_path()
    here = build.calls_path()
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert build.calls_path() != here


@pytest.mark.parametrize("broken", ["no compiler", "another torch"])
def test_without_the_module(monkeypatch, tmp_path, broken):
    path = tmp_path / "_calls.so"
    if broken == "another torch":
        path.write_bytes(b"not a module for this torch")
    monkeypatch.setattr(build, "calls_path", lambda: str(path))
    monkeypatch.setattr(build, "_run", lambda cmd: (_ for _ in ()).throw(RuntimeError("build failed: g++")))
    monkeypatch.setattr(ops, "_calls", None)
    with pytest.warns(RuntimeWarning, match="no native form"):
        calls = ops._native()
    assert calls.mmv(1, 2, 3, 4) is None and calls.linear(1) is None and calls.draft_logits() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert ops._native() is calls       # said once


def test_a_prebuilt_library_is_enough():
    """lib() builds nothing when the library is there, whether the module is or not."""
    code = ("from orin_qwen_lossless_b200 import _lib, build\n"
            "build.calls_path = lambda: '/nonexistent/_calls.so'\n"
            "def no(*a, **k): raise AssertionError('built')\n"
            "build.build = build.build_library = build.build_calls = no\n"
            "_lib.lib()\n")
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT)


def test_the_module_loads():
    m = _lib.calls()
    m.register(ops.Weight, ops.Meta)
    assert m.mmv(None, None, None, None) is None

"""CPU tests of the build and of loading what it built: the extension belongs to one interpreter and one torch, and both are checked."""
import importlib.machinery

import pytest
import torch

from quamba_b200 import _lib, build


def test_the_extension_carries_the_interpreters_tag():
    assert build.NATIVE.name == "_native" + importlib.machinery.EXTENSION_SUFFIXES[0]
    assert build.NATIVE.exists() and not (build.PKG / "_native.so").exists()


def test_an_extension_of_another_torch_is_refused(monkeypatch):
    assert _lib.native().torch_version == torch.__version__
    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    with pytest.raises(RuntimeError, match="built for torch"):
        _lib.native()


def test_objects_are_stale_when_their_command_changes(tmp_path):
    obj, src = tmp_path / "x.cpp.o", build.CSRC / build.NATIVE_SOURCES[0]
    cmd, _ = build._native_flags()
    obj.write_text("")
    assert build._stale(obj, src, cmd)                            # made by nobody knows what
    build._command_file(obj).write_text(" ".join(cmd))
    assert not build._stale(obj, src, cmd)
    assert any(torch.__version__ in c for c in cmd)
    assert build._stale(obj, src, [c.replace(torch.__version__, "9.9.9") for c in cmd])

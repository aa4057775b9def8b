"""What the build does where torch, its headers or a compiler are not there, or are others than before."""
import os
import sys

import pytest

from nvfp4_gemm_b200 import _lib, build


@pytest.fixture
def elsewhere(tmp_path, monkeypatch):
    """An up-to-date C library, no binding yet, and a compiler that only notes what it is asked for."""
    asked = []

    def compile_(target, cmd, verbose):
        asked.append(target.name)
        if target == build.BINDING:
            text = next(c for c in cmd if c.startswith("-DNVFP4_BUILT_FOR="))[len('-DNVFP4_BUILT_FOR="'):-1]
            target.write_bytes(b"\x7fELF nvfp4_native built for: " + text.encode() + b"\0")

    (tmp_path / "libnvfp4_b200.so").write_bytes(b"")
    os.utime(tmp_path / "libnvfp4_b200.so", (2e9, 2e9))
    monkeypatch.setattr(build, "LIB", tmp_path / "libnvfp4_b200.so")
    monkeypatch.setattr(build, "BINDING", tmp_path / "_native.so")
    monkeypatch.setattr(build, "_replace", compile_)
    return asked


@pytest.mark.parametrize("missing", ["torch", "g++"])
def test_the_c_library_is_built_without_torch_or_a_host_compiler(elsewhere, monkeypatch, capsys, missing):
    if missing == "torch":
        monkeypatch.setitem(sys.modules, "torch", None)
    else:
        monkeypatch.setattr(build.shutil, "which", lambda name: None if name == "g++" else "/usr/bin/" + name)
    monkeypatch.setattr(build, "find_nvcc", lambda: "nvcc")
    assert build.build(force=True) == build.LIB
    assert elsewhere == ["libnvfp4_b200.so"] and missing in capsys.readouterr().err
    assert not build.needs_build()


def test_a_binding_of_another_torch_is_built_again_and_not_loaded(elsewhere, monkeypatch):
    build.build()
    assert elsewhere == ["_native.so"] and not build.needs_build()
    os.utime(build.BINDING, (2e9, 2e9))                      # newer than any source
    monkeypatch.setattr(build, "binding_target", lambda: "torch 0.0, C++11 ABI 1, cpython-312-x86_64-linux-gnu")
    assert build.needs_build()
    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.setattr(_lib, "load", lambda: None)
    with pytest.raises(ImportError, match="is built for torch .*this is torch 0.0"):
        _lib.native()
    build.build()
    assert elsewhere == ["_native.so"] * 2 and not build.needs_build()


def test_the_binding_that_is_there_fits(lib):
    assert build.binding_built_for() == build.binding_target()

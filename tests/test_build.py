"""The build's two products depend on different tools: the library (C ABI) must not need what only the host module needs."""
import os
import stat
import sys

import pytest

from vortex_b200 import build


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """The build with its outputs under tmp_path and a compiler that writes its own arguments to its output."""
    nvcc = tmp_path / "nvcc"
    nvcc.write_text('#!/bin/sh\nwhile [ "$1" != -o ]; do shift; done\necho "$@" > "$2"\n')
    nvcc.chmod(nvcc.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setenv("NVCC", str(nvcc))
    monkeypatch.setattr(build, "LIBDIR", str(tmp_path))
    monkeypatch.setattr(build, "OBJDIR", str(tmp_path / "obj"))
    monkeypatch.setattr(build, "LIB", str(tmp_path / "lib.so"))
    monkeypatch.setattr(build, "HOST_LIB", str(tmp_path / "host.so"))
    return tmp_path


def test_library_is_built_without_torch(tree, monkeypatch, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)          # import torch raises
    assert build.build() == str(tree / "lib.so") and os.path.exists(tree / "lib.so")
    assert not os.path.exists(tree / "host.so") and "host module not built" in capsys.readouterr().err


def test_library_is_linked_when_the_host_module_fails(tree, monkeypatch):
    def fail(force):
        raise RuntimeError("g++ failed")

    monkeypatch.setattr(build, "_build_host", fail)
    with pytest.raises(RuntimeError, match="g\\+\\+ failed"):
        build.build()
    assert os.path.exists(tree / "lib.so")


def test_objects_of_an_unfinished_build_are_linked(tree, monkeypatch):
    monkeypatch.setattr(build, "_build_host", lambda force: None)
    build.build()
    os.utime(tree / "lib.so", (1, 1))                         # the library is older than its up-to-date objects
    build.build()
    assert os.path.getmtime(tree / "lib.so") > 1

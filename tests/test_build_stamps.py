"""When tinygpt_b200.build makes what: the library and the torch extension have a stamp each, and the extension's covers the torch and the Python that
it is bound to.  Compilers are replaced by one that records its call and writes the file it was asked for."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from tinygpt_b200 import build


@pytest.fixture
def calls(tmp_path, monkeypatch):
    seen = []

    def run(cmd, **kw):
        seen.append("g++" if cmd[0] == "g++" else "nvcc")
        if seen[-1] == "g++" and made.fails:
            return subprocess.CompletedProcess(cmd, 1, "", "no torch headers")
        Path(cmd[cmd.index("-o") + 1]).write_text("")
        return subprocess.CompletedProcess(cmd, 0, "", "")

    for name, value in dict(LIB_DIR=tmp_path / "lib", OBJ_DIR=tmp_path / "lib/obj", LIB_PATH=tmp_path / "lib/libb200decode.so",
                            NATIVE_PATH=tmp_path / "lib/b200ops.so", SOURCES=["ops.cu"], _nvcc=lambda: "/usr/local/cuda/bin/nvcc").items():
        monkeypatch.setattr(build, name, value)
    monkeypatch.setattr(build.subprocess, "run", run)

    def made():
        seen.clear()
        build.build()
        return sorted(set(seen))

    made.fails = False
    return made


def test_nothing_is_made_twice(calls):
    assert calls() == ["g++", "nvcc"] and calls() == []


@pytest.mark.parametrize("what", ["torch", "python", "abi"])
def test_another_torch_or_python_makes_the_extension_again(calls, monkeypatch, what):
    calls()
    if what == "torch":
        monkeypatch.setattr(torch, "__version__", "9.9")
    elif what == "python":
        monkeypatch.setattr(sys, "version", "9.9")
    else:
        monkeypatch.setattr(torch._C, "_GLIBCXX_USE_CXX11_ABI", not torch._C._GLIBCXX_USE_CXX11_ABI)
    assert calls() == ["g++"] and calls() == []


def test_the_library_is_kept_when_the_extension_fails(calls):
    calls.fails = True
    with pytest.raises(RuntimeError, match="torch_ops"):
        calls()
    calls.fails = False
    assert build.LIB_PATH.exists() and calls() == ["g++"]


def test_a_missing_file_is_made(calls):
    calls()
    build.NATIVE_PATH.unlink()
    assert calls() == ["g++"]
    build.LIB_PATH.unlink()
    assert calls() == ["nvcc"]

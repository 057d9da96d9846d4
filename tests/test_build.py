"""CPU suite: when the Python operators are built again, what is built without a torch, and what the compiler says of the kernels."""
import os
import re
import subprocess
import sys

import pytest

from nacho_b200 import build


@pytest.fixture
def commands(monkeypatch, tmp_path):
    """A tree of its own in which compilers only leave an empty output; yields what was run."""
    ran = []

    def run(cmd, **_):
        ran.append(cmd)
        open(cmd[cmd.index("-o") + 1], "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build.subprocess, "run", run)
    monkeypatch.setattr(build, "NATIVE", str(tmp_path / "_native.so"))
    monkeypatch.setattr(build, "NATIVE_FOR", str(tmp_path / "native.txt"), raising=False)
    return ran


def test_operators_are_built_once_per_interpreter_and_torch(commands, monkeypatch):
    import torch
    nvcc = build._nvcc()
    assert build.build_native(nvcc) == build.NATIVE and len(commands) == 1
    assert build.build_native(nvcc) == build.NATIVE and len(commands) == 1
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    build.build_native(nvcc)
    assert len(commands) == 2
    os.remove(build.NATIVE_FOR)  # built by a version of this file that left no note
    build.build_native(nvcc)
    assert len(commands) == 3
    build.build_native(nvcc)
    assert len(commands) == 3


def test_without_torch_the_library_is_built(commands, monkeypatch, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)
    assert build.build_native(build._nvcc()) is None
    assert not commands and "torch is not installed" in capsys.readouterr().err


def test_fills_of_large_tiles_stay_in_registers():
    """Tiles that fill a room of the result's own length, four CTAs of 64 registers a thread to an SM, hold at most some words more: with
    the columns of all results at once they spilled 80 bytes a thread (220 beside 64-bit keys) and lost what copying the values gains."""
    build.build()
    found = {name: bytes_ for name, bytes_ in build.spills("csr_merge").items() if re.search(r"csr2_tile(_wide)?ILi31ELi0ELi1ELb0E", name)}
    assert len(found) == 2  # 32- and 64-bit keys
    assert all(max(b) <= 64 for b in found.values()), found

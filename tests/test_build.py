"""CPU suite: when the Python operators are built again, and what is built without a torch."""
import os
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

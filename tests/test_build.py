"""CPU suite: what is built without a torch."""
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
    return ran


def test_without_torch_the_library_is_built(commands, monkeypatch, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)
    assert build.build_native(build._nvcc()) is None
    assert not commands and "torch is not installed" in capsys.readouterr().err

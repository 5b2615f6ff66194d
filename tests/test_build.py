"""The same sources give the same code: no flag whose result depends on how a build's work
happens to be spread over threads."""
import subprocess

from fhe_b200 import build


def test_no_source_is_compiled_in_parts(monkeypatch, tmp_path):
    commands = []
    monkeypatch.setattr(build, "BUILD", str(tmp_path))
    monkeypatch.setattr(build, "LIB", str(tmp_path / "lib.so"))

    def run(cmd, check):
        commands.append(cmd)
        open(cmd[cmd.index("-o") + 1], "w").close()

    monkeypatch.setattr(subprocess, "run", run)
    build.build()
    assert sum(c.endswith(".cu") for cmd in commands for c in cmd) >= 15
    assert not [cmd for cmd in commands if any("split-compile" in a for a in cmd)]

"""The incremental build recompiles a source when any header it may include changes,
.h and .cuh alike (run with a stand-in for nvcc)."""
import os
import stat

import pytest

from sar_cambrianaccelerationcard_gb300 import build


@pytest.mark.parametrize("changed", ["a.cu", "b.h", "c.cuh"])
def test_headers_are_dependencies(tmp_path, monkeypatch, changed):
    src, out, log = tmp_path / "csrc", tmp_path / "_build", tmp_path / "log"
    src.mkdir()
    out.mkdir()
    for name in ("a.cu", "b.h", "c.cuh"):
        (src / name).write_text("")
        os.utime(src / name, (1000, 1000))
    nvcc = tmp_path / "nvcc"
    nvcc.write_text(f'#!/bin/sh\necho run >> {log}\nfor o; do last="$o"; done\n: > "$last"\n')
    nvcc.chmod(nvcc.stat().st_mode | stat.S_IEXEC)
    monkeypatch.setenv("NVCC", str(nvcc))
    monkeypatch.setattr(build, "CSRC", str(src))
    monkeypatch.setattr(build, "ROOT", str(tmp_path))
    (tmp_path / "include").mkdir()
    (tmp_path / "include" / "sarbp.h").write_text("")
    os.utime(tmp_path / "include" / "sarbp.h", (1000, 1000))

    def runs():
        build._compile("a.cu", build_dir=str(out))
        return log.read_text().count("run")
    assert runs() == 1 and runs() == 1  # up to date
    os.utime(src / changed, None)
    os.utime(out / "a.o", (2000, 2000))
    assert runs() == 2, changed

"""Objects and library are rebuilt when anything that decides them is newer: a source, a header of either kind, the
public header, or the build file with its per-source flags."""
import importlib.util
import os
from pathlib import Path

import pytest

BUILD = Path(__file__).resolve().parents[1] / "cms-julia_b200" / "build.py"


@pytest.fixture()
def tree(tmp_path, monkeypatch):
    pkg = tmp_path / "pkg"
    (pkg / "csrc").mkdir(parents=True)
    (tmp_path / "include").mkdir()
    (pkg / "build.py").write_text(BUILD.read_text())
    spec = importlib.util.spec_from_file_location("build_under_test", pkg / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    for name in ("csrc/scan.cu", "csrc/k_fit.cu", "csrc/shared.cuh", "csrc/ctx.h"):
        (pkg / name).write_text("")
    (tmp_path / "include" / "pxl.h").write_text("")
    made = []

    def run(cmd, check):
        out = Path(cmd[cmd.index("-o") + 1])
        out.write_text("")
        made.append(out.name)

    monkeypatch.setattr(build.subprocess, "run", run)
    for f in tmp_path.rglob("*"):
        os.utime(f, (1000, 1000))
    build.build_cuda()
    assert sorted(made) == ["k_fit.o", "libpxl_b200.so", "scan.o"]
    made.clear()
    build.build_cuda()
    assert made == []
    return pkg, build, made


@pytest.mark.parametrize("changed,objects", [("csrc/k_fit.cu", {"k_fit.o"}), ("csrc/shared.cuh", {"k_fit.o", "scan.o"}),
                                             ("csrc/ctx.h", {"k_fit.o", "scan.o"}), ("build.py", {"k_fit.o", "scan.o"}),
                                             ("../include/pxl.h", {"k_fit.o", "scan.o"})])
def test_rebuilt(tree, changed, objects):
    pkg, build, made = tree
    later = (pkg / "lib" / "libpxl_b200.so").stat().st_mtime + 100
    os.utime(pkg / changed, (later, later))
    build.build_cuda()
    assert set(made) == objects | {"libpxl_b200.so"}

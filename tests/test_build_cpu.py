"""The build with a stand-in compiler: one library comes out, and a failing build leaves nothing behind."""

from __future__ import annotations

import importlib.util
from pathlib import Path

import pytest

BUILD = Path(__file__).resolve().parents[1] / "challenge-cup_b200" / "build.py"

# writes its inputs' names to -o; fails on a source or object of the name in $FAIL
_NVCC = """#!/bin/sh
out=; inputs=
while [ $# -gt 0 ]; do
  case "$1" in -o) out=$2; shift;; *.cu|*.o) inputs="$inputs $(basename $1)";; esac
  shift
done
echo "$inputs" > "$out"
case "$inputs" in *"$FAIL"*) exit 1;; esac
"""


@pytest.fixture
def build(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("ertm_build_under_test", BUILD)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    nvcc = tmp_path / "cuda" / "bin" / "nvcc"
    nvcc.parent.mkdir(parents=True)
    nvcc.write_text(_NVCC)
    nvcc.chmod(0o755)
    monkeypatch.setenv("CUDA_HOME", str(tmp_path / "cuda"))
    monkeypatch.setenv("FAIL", "none-of-them")
    package = tmp_path / "package"
    package.mkdir()
    mod.OUT = package / "lib.so"
    return mod


def test_build_writes_the_library_alone(build):
    build.build(force=True)
    assert [p.name for p in build.OUT.parent.iterdir()] == ["lib.so"]
    assert build.OUT.read_text().split() == [f"{s.stem}.o" for s in build.SOURCES]


@pytest.mark.parametrize("fail", ["wave.cu", "wave.o"])
def test_failed_build_leaves_the_package_as_it_was(build, monkeypatch, fail):
    build.OUT.write_text("earlier build")
    monkeypatch.setenv("FAIL", fail)
    with pytest.raises(RuntimeError):
        build.build(force=True)
    assert [p.name for p in build.OUT.parent.iterdir()] == ["lib.so"]
    assert build.OUT.read_text() == "earlier build"

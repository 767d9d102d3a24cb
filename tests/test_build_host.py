"""The build on a host without a GPU: what it needs, and what it leaves behind.  The compilers are stand-ins."""
import importlib.util
import os
import stat

import pytest

from llm170_b200 import build

FAKE_NVCC = """#!/bin/sh
out=
for a in "$@"; do
  case "$a" in *{bad}*) if [ -n "{bad}" ]; then echo no; exit 1; fi;; esac
  if [ "$prev" = "-o" ]; then out="$a"; fi
  prev="$a"
done
echo made > "$out"
"""


@pytest.fixture
def sandbox(tmp_path, monkeypatch):
    for name in ("SO", "HASH", "NATIVE_SO", "NATIVE_HASH"):
        monkeypatch.setattr(build, name, str(tmp_path / os.path.basename(getattr(build, name, name))), raising=False)

    def nvcc(bad=""):
        path = tmp_path / "nvcc"
        path.write_text(FAKE_NVCC.replace("{bad}", bad))
        path.chmod(path.stat().st_mode | stat.S_IXUSR)
        monkeypatch.setenv("NVCC", str(path))

    return tmp_path, nvcc


def test_the_library_builds_where_torch_is_not_installed(sandbox, monkeypatch):
    tmp_path, nvcc = sandbox
    nvcc()
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    so = build.build(force=True)
    assert open(so).read() == "made\n"
    assert not (tmp_path / "_native.so").exists()
    os.remove(tmp_path / "nvcc")
    assert build.build() == so                     # current: nothing is compiled again


def test_a_failed_build_leaves_nothing_behind(sandbox):
    tmp_path, nvcc = sandbox
    nvcc(bad="head.cu")
    before = sorted(os.listdir(build.CSRC))
    with pytest.raises(RuntimeError, match="head.cu"):
        build.build(force=True)
    assert sorted(os.listdir(build.CSRC)) == before
    assert sorted(os.listdir(tmp_path)) == ["nvcc"]

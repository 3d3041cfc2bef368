"""Host-side pieces of the native libraries that need no GPU."""
import fnmatch
import subprocess
import sys
import tomllib
from pathlib import Path

import pytest

import dcp_b200
from dcp_b200.csrc import build
from dcp_b200.ops import _lib

FAKE_RUNTIME = r"""
#include <cstdio>
#include <initializer_list>
#include "smem_limit.h"
static int device = 0, raised_on[70] = {}, fail = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  if (fail) return cudaErrorInvalidValue;
  ++raised_on[device];
  return cudaSuccess;
}
static void kernel() {}
int main() {
  std::atomic<uint64_t> raised{0};
  fail = 1;
  if (dcpk::raise_smem_limit(kernel, 200000, raised) == cudaSuccess) return 1;   // a refusal is reported, and asked again
  fail = 0;
  for (int d : {0, 1, 0, 1, 63, 63, 0, 64, 64}) {
    device = d;
    if (dcpk::raise_smem_limit(kernel, 200000, raised) != cudaSuccess) return 2;
  }
  std::printf("%d %d %d %d\n", raised_on[0], raised_on[1], raised_on[63], raised_on[64]);
}
"""


def test_shared_memory_limit_is_raised_once_on_each_device(tmp_path):
    """Against a fake runtime: the limit belongs to a device, so a kernel's first launch on a second one raises it again."""
    src, exe = tmp_path / "fake.cpp", tmp_path / "fake"
    src.write_text(FAKE_RUNTIME)
    cuda = Path(build._nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-I%s" % build.KERNEL_DIR, "-I%s" % cuda, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, stdout=subprocess.PIPE, text=True).stdout.split() == ["1", "1", "1", "2"]


def test_package_data_holds_every_native_source():
    """An installed copy can rebuild all of its libraries."""
    patterns = tomllib.loads((build.PKG.parent / "pyproject.toml").read_text())["tool"]["setuptools"]["package-data"]["dcp_b200"]
    sources = [p.relative_to(build.PKG).as_posix() for p in build.HERE.rglob("*") if p.suffix in (".cu", ".cuh", ".h", ".hpp", ".cpp")]
    assert len(sources) > 20 and [s for s in sources if not any(fnmatch.fnmatch(s, p) for p in patterns)] == []


def test_build_of_an_incomplete_copy_says_so(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "HOST_DIR", tmp_path)
    with pytest.raises(RuntimeError, match="incomplete"):
        build.build_calls(force=True)


def test_missing_and_unloadable_native_calls_are_told_apart(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "load", lambda: None)
    monkeypatch.setattr(_lib, "calls_path", lambda: tmp_path / "_calls.so")
    monkeypatch.delattr(dcp_b200, "_calls", raising=False)
    monkeypatch.setitem(sys.modules, "dcp_b200._calls", None)      # the import fails
    with pytest.raises(RuntimeError, match="missing"):
        _lib.calls()
    (tmp_path / "_calls.so").touch()
    with pytest.raises(RuntimeError, match="does not load"):
        _lib.calls()

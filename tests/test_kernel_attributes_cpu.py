"""CPU: a kernel's shared-memory attribute and its residency are set and asked for
once on every device a process launches it on, not once per process (the host
helpers of csrc/attr.h, compiled against a CUDA runtime that counts the calls)."""
import os
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include "attr.h"
#include <cstdio>
#include <map>
#include <tuple>
static int device = 0, failing = 0;
static std::map<std::tuple<const void*, int, int>, int> set;   // kernel, device, attribute
static std::map<std::pair<const void*, int>, int> asked;       // kernel, device
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int) {
  if (failing) return cudaErrorInvalidValue;
  set[{f, device, (int)a}]++;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int d) { *v = 100 + d; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t, unsigned) {
  asked[{f, device}]++;
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int, size_t) {
  asked[{f, device}]++;
  *n = 2;
  return cudaSuccess;
}
}
static void one(int) {}
static void two(int) {}
int bad = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); bad = 1; } } while (0)
int main() {
  bcmg::SharedMemory a, b;
  bcmg::Resident r;
  const int smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  failing = 1;
  CHECK(a.allow(one, 100000) == cudaErrorInvalidValue);
  failing = 0;
  for (int round = 0; round < 3; round++)
    for (device = 0; device < 70; device++) {
      CHECK(a.allow(one, 100000) == cudaSuccess);
      CHECK(b.allow(two, 100000) == cudaSuccess);
      int n = 0;
      CHECK(r.ctas(one, 256, 100000, &n) == cudaSuccess && n == 2 * (100 + device));
    }
  for (int d = 0; d < 70; d++) {
    const int want = d < 64 ? 1 : 3;
    CHECK((set[{(const void*)one, d, smem}] == want && set[{(const void*)two, d, smem}] == want));
    CHECK((asked[{(const void*)one, d}] == want));
  }
  return bad;
}
"""


def test_set_once_per_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = Path(os.path.realpath(nvcc)).parents[1] / "include"
    if not (inc / "cuda_runtime.h").exists() or not shutil.which("g++"):
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "bcmtools_gb300" / "csrc"), "-I", str(inc),
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_launchers_keep_no_flag_of_their_own():
    for p in (ROOT / "bcmtools_gb300" / "csrc").iterdir():
        if p.suffix in (".cu", ".cuh"):
            found = re.findall(r"^\s+static (?:bool|int) \w+(?:\[\d+\])? *=.*", p.read_text(), re.M)
            assert not found, (p.name, found)

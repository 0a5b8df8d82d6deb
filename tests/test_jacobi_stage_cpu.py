"""CPU: the fused Jacobi sweep's stage leaves as many CTAs of 16^3 blocks on an SM (228
KB of shared memory, 1 KB of it per CTA) as the block's brick and b's interior planes
alone would: two in FP64."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include "stage.cuh"
#include <cstdio>
template <typename T, int N, int VC> void show() {
  std::printf("%d %d %d %zu\n", (int)sizeof(T), N, VC, bcmg::BrickStage<T, N, VC, true>::SMEM);
}
int main() {
  show<float, 8, 1>(); show<float, 8, 2>(); show<float, 16, 1>(); show<float, 16, 2>();
  show<double, 8, 1>(); show<double, 8, 2>(); show<double, 16, 1>(); show<double, 16, 2>();
}
"""


def test_stage_holds_what_the_sweep_needs(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("needs nvcc")
    (tmp_path / "t.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    str(ROOT / "include"), "-I", str(ROOT / "bcmtools_gb300" / "csrc"), str(tmp_path / "t.cu"),
                    "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout
    ctas = {}
    for line in out.splitlines():
        es, n, vc, smem = (int(x) for x in line.split())
        lx = n + 2 * vc
        most = 233472 // (16 + (lx ** 3 + n * lx * lx) * es + 1024)
        ctas[es, n, vc] = 233472 // (smem + 1024)
        assert ctas[es, n, vc] == most or (es, n, vc) == (8, 8, 1), line  # 13 of 64 threads, not 15
    assert ctas[8, 16, 2] == 2

"""The host-side rules that choose launch shapes (tri_step_launch.h), compiled
and run on the CPU."""
import os
import shutil
import subprocess

import pytest

from triton_b200 import build

PROGRAM = r"""
#include <cstdio>
#include "tri_step_launch.h"
int main() {
  // FP32 batches of square members: cells in all -> budget, height
  for (double cells : {1.0e6, 2.6e6, 6.0e6, 16.3e6, 263e6}) {
    const tri::FluxShape s = tri::flux_shape(false, true, 1.0, [&](int rb) { return (long)(cells / 30 / rb); });
    std::printf("%d %d ", s.variant, s.rb);
  }
  std::printf("\n");
}
"""


def test_fp32_batch_budget_by_tile_height(tmp_path):
    """Short tiles (small batches) take 6 blocks per SM, those of 12 rows and
    more 8: measured on batches of 9 to 256 members."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "shapes.cu", tmp_path / "shapes"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "--fmad=false", "-I" + build.CSRC,
                    "-I" + os.path.join(build.ROOT, "include"), "-o", str(exe), str(src)], check=True)
    got = [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    shapes = list(zip(got[::2], got[1::2]))
    assert [v for v, _ in shapes] == [1, 1, 2, 2, 2] and [rb >= 12 for _, rb in shapes] == [False, False, True, True, True]

"""CPU test of the rule that lets the strict-FP32 convolution decode its reduction indices through a table: an entry beyond the
reduction may not lead to a row of the image, wherever the padding puts the output's first and last rows."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "conv_fp32_table.h"
#include <cstdio>
using namespace gieb;
int main() {
  const int kernels[] = {1, 3, 7, 300};
  const int heights[] = {1, 56, 32000, 32500, 32700, 32760, 32764, 32765, 32766, 32767, 32768, 33000, 40000};
  const int pads[] = {0, 1, 2, 3, 20, 67, 100, 300, 1000, 32766, 32767, 70000, 2147483647};
  long accepted = 0, bad = 0;
  for (int r : kernels) for (int h : heights) for (int pad : pads) {
    if (!conv_fp32_table_fits(16, 4, h, 3, r, 1, pad)) continue;
    ++accepted;
    const long rows = long(h) + 2L * pad - r + 1;  // input rows of the filter's first tap: -pad .. -pad + rows - 1
    for (long oh = 0; oh < rows; ++oh) {
      const long ih = oh - pad + kNoRow;
      if (ih >= 0 && ih < h) { ++bad; if (bad < 5) std::printf("h %d pad %d r %d: output row %ld reads row %ld\n", h, pad, r, oh, ih); break; }
    }
  }
  std::printf("%ld accepted, %ld bad\n", accepted, bad);
  if (!conv_fp32_table_fits(4096, 64, 56, 56, 3, 3, 1) || conv_fp32_table_fits(4097, 64, 56, 56, 3, 3, 1)) return 2;
  if (!conv_fp32_table_fits(16, 2, 32700, 1, 3, 1, 67)) return 3;
  return bad != 0 || accepted == 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_entries_beyond_the_reduction_never_read(tmp_path):
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "cuda-inference_b200", "csrc"), str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

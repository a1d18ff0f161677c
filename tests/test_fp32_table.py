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


WIDE_PROGRAM = r"""
#include "conv_fp32_table.h"
#include <cstdio>
using namespace gieb;
int main() {
  // {c, h, w, r, s}: images of up to 2^31 - 1 values, windows that reach into the padding
  const int shapes[][5] = {{64, 56, 56, 3, 3}, {3243932, 2, 331, 3, 3}, {3243933, 2, 331, 3, 3}, {1, 1, 2147483646, 3, 3}, {1, 1, 2147483646, 1, 1}, {2147483647, 1, 1, 1, 1},
                           {64, 5792, 5792, 5, 5}, {1, 1, 200000000, 31, 1}, {1, 46340, 46341, 1, 31}, {16777215, 128, 1, 3, 3}, {2097152, 1, 1023, 3, 5}};
  int accepted = 0, refused = 0, bad = 0;
  for (const auto& d : shapes) {
    long long most = 0;
    for (int r = 0; r < d[3]; ++r)
      for (int s = 0; s < d[4]; ++s) {
        const long long offset = ((d[0] - 1LL) * d[1] + r) * d[2] + s;  // the last channel's
        if (offset > most) most = offset;
      }
    const bool fits = conv_fp32_wide_offsets_fit(d[0], d[1], d[2], d[3], d[4]);
    ++(fits ? accepted : refused);
    if (fits != (most <= 2147483647LL)) { ++bad; std::printf("c %d h %d w %d r %d s %d: largest offset %lld\n", d[0], d[1], d[2], d[3], d[4], most); }
  }
  std::printf("%d accepted, %d refused, %d bad\n", accepted, refused, bad);
  return bad != 0 || accepted < 3 || refused < 3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_offsets_of_the_wide_kernel_fit_32_bits(tmp_path):
    src, exe = tmp_path / "wide.cpp", tmp_path / "wide"
    src.write_text(WIDE_PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "cuda-inference_b200", "csrc"), str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_wide_tiles_leave_images_whose_offsets_do_not_fit(pkg):
    """One channel more than fits, and the kernel that indexes in 64 bits takes the layer (tiles of 64 pixels instead of 128)."""
    tiles = [pkg.query(pkg.ConvProblem(8, c, 2, 331, 64, 3, 3, 1, 1, 1, 1, precision=pkg.FP32)).cfg.tile_m for c in (3243932, 3243933)]
    assert tiles == [128, 64]


SLABS_PROGRAM = r"""
#include "conv_fp32_table.h"
int main() {
  const int ks[] = {1, 15, 16, 17, 576, 2147483631, 2147483632, 2147483633, 2147483647};
  for (int k : ks) if (gieb::fp32_slabs(k) != int((k + 15LL) / 16)) return 1;
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_slabs_of_the_longest_reductions(tmp_path):
    src, exe = tmp_path / "slabs.cpp", tmp_path / "slabs"
    src.write_text(SLABS_PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "cuda-inference_b200", "csrc"), str(src), "-o", str(exe)])
    assert subprocess.run([str(exe)]).returncode == 0

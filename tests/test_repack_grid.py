"""CPU test of the repack grids: planes and channel counts within a tile of 2^31 get the tiles that they have."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "repack_grid.h"
#include <cstdio>
#include <initializer_list>
using namespace gieb;
int main() {
  int bad = 0;
  const int tiles[] = {32, 64, 128};
  for (int tile : tiles)
    for (long long n : {1LL, tile - 1LL, tile + 0LL, tile + 1LL, 2147483520LL, 2147483583LL, 2147483584LL, 2147483616LL, 2147483644LL, 2147483646LL, 2147483647LL}) {
      const long long want = n / tile + (n % tile != 0);
      if (tiles_of(int(n), tile) != want) { ++bad; std::printf("%lld elements in tiles of %d: %d\n", n, tile, tiles_of(int(n), tile)); }
    }
  // a source on every boundary; runs of 4, 2 and 1 pixels
  const struct { int hw; unsigned long src; int pixels; } rows[] = {{2147483644, 256, 4}, {2147483644, 260, 2}, {2147483644, 258, 1}, {2147483646, 256, 2}, {2147483647, 256, 1}, {196, 8, 4}, {198, 8, 2}, {199, 8, 1}};
  for (const auto& r : rows) {
    const int v = direct_pixels(r.hw, r.src);
    const long long blocks = direct_blocks(v, r.hw, 72, 3), want = ((long long)r.hw + 32 * v - 1) / (32 * v) * 2 * 3;
    if (v != r.pixels || blocks != want) { ++bad; std::printf("plane of %d at %lu: %d pixels, %lld blocks\n", r.hw, r.src, v, blocks); }
  }
  return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_tiles_of_the_largest_planes(tmp_path):
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-ftrapv", "-I" + os.path.join(ROOT, "cuda-inference_b200", "csrc"), str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_every_repack_asks_whether_to_prefetch():
    """GIEB_DISABLE_PREFETCH switches the fills ahead of the dependency wait off in every file that issues them there."""
    csrc = os.path.join(ROOT, "cuda-inference_b200", "csrc")
    texts = {f: open(os.path.join(csrc, f)).read() for f in sorted(os.listdir(csrc)) if f.startswith("repack") and f.endswith(".cu")}
    issuing = [f for f, t in texts.items() if "prefetch_l2(" in t]
    assert len(issuing) == 2
    for f in issuing:
        assert "prefetch_enabled()" in texts[f], f

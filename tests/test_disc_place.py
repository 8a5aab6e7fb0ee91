"""Places of overflowing disc lists in their pool, which may hold more than 2^32
entries: a round trip on the CPU through the header that the kernels use, and
that both kernels go through it."""

import os
import subprocess

from bone_morphometry_gb300 import build

PROGRAM = r"""
#include <cstdio>
#include "disc_place.h"
int main() {
  const unsigned long long places[] = {0ull, 4ull, 0xfffffffcull, 0x100000000ull, 0x100000004ull, 9332000000ull,
                                       0x3fffffffcull};
  for (unsigned long long p : places)
    if (bm::disc_first(bm::disc_place(p)) != p) return 1;
  // segments keep the next place a multiple of 4, and hold their list
  for (unsigned n = 1; n < 70000; ++n)
    if (bm::disc_segment(n) % 4 != 0 || bm::disc_segment(n) < n || bm::disc_segment(n) > n + 3) return 2;
  return 0;
}
"""


def test_places_beyond_32_bits(tmp_path):
    src = tmp_path / "places.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "places")
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_kernels_keep_the_place_whole():
    text = open(os.path.join(build.CSRC, "discs.cu")).read()
    assert "disc_place(first)" in text and "disc_first(__ldg(&list->x))" in text
    assert "(uint32_t)first" not in text and "disc_segment(cnt)" in text

"""The counting sort's slices, up to the largest batch that an entry takes:
they cover the points once, in order, and nothing on the way leaves its
type (compiled for the host with the undefined-behaviour checks on)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <limits.h>
#include <stdio.h>
#include "sort_slices.h"
int main() {
  const int64_t sizes[] = {1, 2, 15, 16, 17, 65535, 131072, 131073, 3000001, INT_MAX - 4096LL, INT_MAX - 127LL,
                           INT_MAX - 1LL, INT_MAX};
  const int counts[] = {16, 17, 127, 128};
  for (int64_t n : sizes)
    for (int blocks : counts) {
      int64_t at = 0;
      for (int b = 0; b < blocks; b++) {
        const eg::SortSlice s = eg::sort_slice(n, b, blocks);
        if (s.lo != at || s.hi < s.lo || s.hi > n) return 1;
        const int lanes[] = {0, 1023};
        for (int tid : lanes) {  // a thread's points, from near the slice's end
          auto p = s.lo + tid;
          while (p + 1024 < s.hi - 4096) p += (s.hi - 4096 - p) / 1024 * 1024;
          for (; p < s.hi; p += 1024)
            if (p < s.lo) return 2;
          if (p < s.lo) return 3;
        }
        at = s.hi;
      }
      if (at != n) return 4;
    }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_slices_cover_the_largest_batches(tmp_path):
    src, exe = tmp_path / "slices.cc", tmp_path / "slices"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-fsanitize=undefined",
                    "-fno-sanitize-recover=undefined", "-I", os.path.join(ROOT, "einspline_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)

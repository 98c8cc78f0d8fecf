"""Staging buffers of the projection kernel's epilogue (csrc/linear.cuh): a buffer is written again only when the copy
that reads it is none of the warp's last kStoreBufs - 1, which are all that its wait lets be under way."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mini-attention_b200" / "csrc"
CUDA = Path("/usr/local/cuda/include")

# Every tile width, up to six tiles of a warp, each whole or cut short by the weight's last column.
WALK = r"""
#include <cuda_runtime.h>
#include "linear.cuh"
#include <cstdio>
int main() {
  int walks = 0;
  for (int bn = 16; bn <= ma::kLinearMaxBn; bn += 16)
    for (int half = 0; half < 2; ++half)
      for (int cut = 0; cut < bn; cut += 16)          // columns that every second tile lacks
        for (int tiles = 1; tiles <= 6; ++tiles, ++walks) {
          int used_by[ma::kStoreBufs], copies = 0;    // which copy a buffer was last read by
          for (int& u : used_by) u = -1;
          ma::StoreTurn turn;
          for (int t = 0; t < tiles; ++t)
            for (int bx = half; bx < bn / 16 && bx * 16 < bn - (t & 1) * cut; bx += 2) {
              const int at = turn.take();
              if (at < 0 || at >= ma::kStoreBufs) return 1;
              if (used_by[at] >= 0 && used_by[at] > copies - 1 - (ma::kStoreBufs - 1)) return 2;
              used_by[at] = copies++;
            }
        }
  std::printf("%d\n", walks);
  return 0;
}
"""


@pytest.mark.skipif(not (CUDA / "cuda.h").exists(), reason="no CUDA headers")
def test_a_buffer_is_free_before_it_is_written(tmp_path):
    src = tmp_path / "walk.cpp"
    src.write_text(WALK)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", f"-I{CUDA}", str(src), "-o", str(tmp_path / "walk")], check=True)
    r = subprocess.run([str(tmp_path / "walk")], capture_output=True, text=True)
    assert r.returncode == 0 and int(r.stdout) > 1000

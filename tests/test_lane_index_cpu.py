"""Instances that the multiply and divide lane kernels' threads take, from the
header's own function compiled for the host: every instance of a batch whose
threads pass 2^32 is reached once, at the grid that the launchers ask for."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "xmp_b200", "csrc")

CHECK = r"""
#include "lanes.cuh"
#include <cstdio>
using namespace xmpb;
// The first and last thread of blocks about each multiple of 2^32 threads, and of the grid's ends.
template <int TPI> static int check(uint64_t count, int threads) {
  const int64_t grid = grid_for(count * TPI, threads);
  if (grid * threads < (int64_t)(count * TPI) || (grid - 1) * threads >= (int64_t)(count * TPI)) return 1;
  for (uint64_t wrap = 0; wrap <= count * TPI; wrap += 1ull << 32)
    for (int64_t at = (int64_t)(wrap / threads) - 2; at <= (int64_t)(wrap / threads) + 2; at++)
      for (int64_t b : {at, grid - 1 - (int64_t)(wrap >> 32)})
        if (b >= 0 && b < grid)
          for (uint64_t t : {0ull, 1ull, threads - 1ull})
            if (lane_instance<TPI>((uint32_t)b, threads, (uint32_t)t) != ((unsigned __int128)b * threads + t) / TPI) return 2;
  return lane_instance<TPI>((uint32_t)(grid - 1), threads, threads - 1) < count - 1 ? 3 : 0;
}
template <int TPI> static int all() {
  int bad = 0;
  for (uint64_t count : {1ull, 37ull, 1ull << 20, (1ull << 32) / TPI - 1, (1ull << 32) / TPI, (1ull << 32) / TPI + 1,
                         (5ull << 30) / TPI + 77})
    for (int threads : {32, 64, 128, 256})
      if (count < 1ull << 32) bad |= check<TPI>(count, threads);
  return bad;
}
int main() {
  printf("%d %d %d %d %d\n", all<2>(), all<4>(), all<8>(), all<16>(), all<32>());
  return 0;
}
"""


def test_every_instance_is_reached(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = str(tmp_path / "check.cu"), str(tmp_path / "check")
    with open(src, "w") as f:
        f.write(CHECK)
    p = subprocess.run([nvcc, "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), src, "-o", exe],
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split() == ["0"] * 5


@pytest.mark.parametrize("source,kernel", [("mul.cu", "mul_lanes_kernel"), ("div.cu", "divmod_lanes_kernel")])
def test_kernels_take_it(source, kernel):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    body = text[text.index("void __launch_bounds__(256) " + kernel):]
    body = body[:body.index("\n}\n")]
    assert re.search(r"uint64_t local = lane_instance<TPI>\(blockIdx.x, blockDim.x, threadIdx.x\)", body)
    assert not re.search(r"uint32_t \w+ = \(?blockIdx.x \* blockDim.x", body)

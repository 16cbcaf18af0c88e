"""Pointer jumping's survivor lists hold every block's region (CPU only: a host program built
against the library's headers).

A block of the sssp kernel writes the vertices that jump again from block * span on, span =
ceil(n / blocks).  In a later round `total` entries are dealt vspan = ceil(total / blocks) to a
block, and a block keeps at most those, so its region is used up to block * span + (its entries).
With vspan < span the last blocks' regions start near, and end past, n.
"""
import os
import shutil
import subprocess

import pytest

from dyng_b200 import build as B

PROGRAM = r"""
#include "internal.hpp"
#include <cstdio>
int main() {
  using namespace dyngb200;
  long long worst = 0;
  for (long long n = 1; n <= 3000; ++n)
    for (long long blocks = 1; blocks < kPjMaxBlocks; blocks += blocks < 8 ? 1 : 7) {
      const long long span = (n + blocks - 1) / blocks;
      for (long long vspan = 1; vspan <= span; ++vspan) {
        const long long total = vspan * blocks < n ? vspan * blocks : n;  // the most with this vspan
        const long long last = (total - 1) / vspan;  // the last block with entries
        const long long end = last * span + (total - last * vspan);
        if (end - n > worst) worst = end - n;
        if (end > pj_list_entries(n)) {
          std::printf("n %lld blocks %lld total %lld: %lld\n", n, blocks, total, end);
          return 1;
        }
      }
    }
  std::printf("%lld\n", worst);
  return 0;
}
"""


def test_regions_fit_their_lists(tmp_path):
    nvcc = B.NVCC if os.path.exists(B.NVCC) else shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("nvcc not found")
    src, exe = tmp_path / "regions.cu", tmp_path / "regions"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O1", "-I", B.CSRC, "-I", os.path.join(B.ROOT, "include"),
                    "--expt-relaxed-constexpr", *B.ARCH, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout) > 0  # regions do end past n

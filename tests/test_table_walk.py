"""The walk over the explicit local matrix's items (a row of the matrix and a part
of a column each), compiled for the host: every item once, also past 2^31 of them."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
PROGRAM = r"""
#include <cstdio>
#include "ttb_device.cuh"
// the entries that ``threads`` walkers visit of rows x width, and whether each is its own
static bool covers(long long rows, int width, int threads, bool all) {
  long long seen = 0;
  for (int t = 0; t < threads; t += all ? 1 : threads - 1) {
    long long e = t;
    for (ttb::TableWalk w(t, threads, width); w.row < rows; w.next(), e += threads, ++seen)
      if (w.row != e / width || w.at != e % width) return false;
    if (e < rows * width) return false;
  }
  return !all || seen == rows * width;
}
int main() {
  const int widths[] = {1, 7, 255, 256, 257, 1000, 2048, 5000};
  for (int w : widths)
    for (int threads : {256, 2048})
      if (!covers(37, w, threads, true)) return 1;
  // a system of 65536 unknowns whose left bond is 1: 2^32 items
  if (!covers(65536, 65536, 2048, false)) return 2;
  std::puts("ok");
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_walk_visits_every_item_once(tmp_path):
    (tmp_path / "walk.cu").write_text(PROGRAM)
    exe = tmp_path / "walk"
    subprocess.run([NVCC, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "ttnumpy_b200/csrc"),
                    "-I", os.path.join(ROOT, "include"), "-o", str(exe), str(tmp_path / "walk.cu")],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok"

"""The row segments and edge lists of the two-way deposit (csrc/deposit_rows.cuh), on the host: for
every row length up to a few segments, every cell takes what its two home cells hold from the lists
of its segment exactly once."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INC = "/usr/local/cuda/include"

SRC = r"""
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdio>
#include "launch.h"
using namespace ch4;
int main() {
  long bad = 0;
  for (int NX = 1; NX < 1300; NX++) {
    const RowSegs g = row_segs(NX);
    const int ns = g.n, len = g.len;
    // no segment empty, none beyond what a warp's shared memory holds
    if ((ns - 1) * len >= NX || ns * len < NX || len > ROW_SEG || (row_places(g) > 1) != (ns > 1)) bad++;
    for (int hx = 0; hx <= NX; hx++) {
      const int b = row_bin(hx, 0, 0, g, 1), e = row_edge_bin(hx, 0, 0, g, 1);
      if (b < 0 || b >= ns || e >= (int)row_lists(g) || (e >= 0 && e < ns)) bad++;
      if (row_bin(hx, 4, 3, g, 4) >= (int)row_bins(g, 4, 3)) bad++;
    }
    for (int seg = 0; seg < ns; seg++) {
      const int x0 = seg * len, n = std::min(len, NX - x0);
      for (int x = x0; x < x0 + n; x++)
        for (int corner = 0; corner < 2; corner++) {
          const int hx = x + corner;  // the home cell whose corner `corner` is x
          int hits = row_seg(hx, g) == seg;
          if (seg + 1 < ns && row_edge_bin(hx, 0, 0, g, 1) == ns + seg) hits++;
          if (hits != 1) bad++;
        }
    }
  }
  std::printf("%ld\n", bad);
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")), reason="no CUDA headers")
def test_every_home_is_met_once(tmp_path):
    src, exe = tmp_path / "rows.cpp", tmp_path / "rows"
    src.write_text(SRC)
    csrc = os.path.join(os.path.dirname(HERE), "ch4-project_b200", "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CUDA_INC, "-I", csrc, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.strip() == "0"

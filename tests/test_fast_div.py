"""fast_div of csrc/lattice.cuh against integer division (the cell coordinates of the step
kernel): every divisor near a power of two, at the multiples of the divisor and one below
them, up to the largest cell index 2^31 - 1."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cuda_runtime.h>
#include "lattice.cuh"
#include <cstdio>
int main() {
  const uint32_t top = 0x7fffffffu;
  for (int e = 0; e <= 30; e++)
    for (int o = -3; o <= 3; o++) {
      const long long dl = (1ll << e) + o;
      if (dl < 1) continue;
      const uint32_t d = (uint32_t)dl;
      const ch4::FastDiv f = ch4::fast_div_of(d);
      const uint32_t q = top / d, step = q / 4096 + 1;
      for (uint64_t k = 0; k <= q; k += step)
        for (long long n : {(long long)(k * d), (long long)(k * d) - 1, (long long)(k * d) + d - 1, (long long)top})
          if (n >= 0 && n <= (long long)top && ch4::fast_div((uint32_t)n, f) != (uint32_t)n / d) {
            std::printf("%lld / %u\n", n, d);
            return 1;
          }
    }
  for (uint32_t d = 1; d < 3000; d++) {
    const ch4::FastDiv f = ch4::fast_div_of(d);
    for (uint32_t k = 0; k < 200; k++)
      for (uint32_t n : {k * d, k * d + d - 1, top - k, top / d * d - (k ? 1u : 0u)})
        if (ch4::fast_div(n, f) != n / d) return 1;
  }
  return 0;
}
"""


def test_fast_div(tmp_path):
    src = tmp_path / "fast_div.cpp"
    src.write_text(DRIVER)
    exe = str(tmp_path / "fast_div")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(REPO, "ch4-project_b200", "csrc"), "-I",
                    "/usr/local/cuda/include", str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0

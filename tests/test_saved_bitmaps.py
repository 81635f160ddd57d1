"""CPU: how many bitmaps of heavy rows are kept between the phases (csrc/cas_workspace.h), compiled as plain C++.

The choice equals the formula that always knows the free memory, for rows, slices, shares and free memory over their
ranges; where 8 GiB hold every bitmap the free memory is not asked for."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "contention-aware-spgemm_b200", "csrc")

HARNESS = r"""
#include "cas_workspace.h"
#include <cmath>
#include <cstdio>
#include <random>

int main() {
  std::mt19937_64 rng(5);
  auto upto = [&](double a, double b) { return std::exp(std::uniform_real_distribution<double>(std::log(a), std::log(b))(rng)); };
  const double gib = 1024.0 * 1024 * 1024;
  int asked = 0, differ = 0, needless = 0;
  for (int i = 0; i < 200000; ++i) {
    const int64_t rows = (int64_t)upto(1, 3e7), slices = (int64_t)upto(1, 4096);
    const double share = i % 3 ? 1.0 : 0.25, free_b = i % 7 ? upto(1e6, 2e11) : 0.0;
    int calls = 0;
    const cas::SavedBitmaps got = cas::saved_bitmaps(rows, slices, 65536, share, [&] { ++calls; return free_b; });
    const double cap = share * std::max(8.0 * gib, std::min(24.0 * gib, 0.25 * free_b));
    const int want = (double)rows * (double)slices * 65536 <= cap ? (int)slices : 1;
    differ += got.slices != want || got.any != ((double)rows * want * 65536 <= cap);
    needless += calls > 1 || (calls && (double)rows * (double)slices * 65536 <= share * 8 * gib);
    asked += calls;
  }
  printf("%d %d %d\n", differ, needless, asked);
  return differ || needless || !asked;
}
"""


def test_choice(tmp_path):
    (tmp_path / "t.cpp").write_text(HARNESS)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-I", CSRC, "-o", str(tmp_path / "t"),
                    str(tmp_path / "t.cpp")], check=True)
    p = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout + p.stderr

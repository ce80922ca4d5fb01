"""csrc/conv_rows.h, the rows that a CTA of the short convolution takes: no split costs less by the rule's own measure, and the search stays short (below a microsecond on
an idle machine, twice that allowed; one through 1024 splits takes 11)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "evo_b200", "csrc")
PROGRAM = r'''
#include "conv_rows.h"
#include <chrono>
#include <cmath>
#include <cstdio>
#include <random>
static int64_t cost(int64_t L, int64_t per, int64_t slots, int64_t rows) { return (per * ((L + rows - 1) / rows) + slots - 1) / slots * (rows + 16); }
int main() {
  std::mt19937_64 rng(7);
  const auto log_uniform = [&](double top) { return std::max<int64_t>(1, (int64_t)std::exp(std::uniform_real_distribution<>(0, std::log(top))(rng))); };
  for (int i = 0; i < 20000; ++i) {
    const int64_t L = log_uniform(131073), per = log_uniform(i % 3 ? 3000 : 70000), slots = 4 * (i % 5 ? 148 : 1 + (int64_t)(rng() % 160)), rows = evo::conv_rows(L, per, slots, 32);
    if (rows < 32 || rows % 4 || rows > std::max<int64_t>(32, (L + 3) / 4 * 4)) { printf("L %ld per %ld: %ld rows\n", (long)L, (long)per, (long)rows); return 1; }
    int64_t least = cost(L, per, slots, rows);
    for (int64_t n = 1; n <= 1024 && (n == 1 || L / n >= 32); ++n) least = std::min(least, cost(L, per, slots, std::max<int64_t>(32, ((L + n - 1) / n + 3) / 4 * 4)));
    if (least < cost(L, per, slots, rows)) { printf("L %ld per %ld slots %ld: %ld rows\n", (long)L, (long)per, (long)slots, (long)rows); return 1; }
  }
  volatile int64_t sum = 0;
  double slowest = 0;
  const int64_t sizes[][2] = {{100, 12}, {4096, 48}, {8193, 12}, {32768, 1}, {8192, 1777}, {131072, 1}, {131072, 48}, {131072, 583}, {1000003, 12}, {1000003, 48}};      // rows, and pairs of 512 channels
  for (const auto& s : sizes) {
    double best = 1e9;
    for (int batch = 0; batch < 50; ++batch) {                                  // the best of many: other work on the machine
      const auto t = std::chrono::steady_clock::now();
      volatile int64_t L = s[0];
      for (int i = 0; i < 100; ++i) sum = sum + evo::conv_rows(L, s[1], 592, 32);
      best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count() * 1e4);
    }
    slowest = std::max(slowest, best);
  }
  printf("%s %.3f us\n", slowest < 2.0 ? "OK" : "SLOW", slowest);
  return 0;
}
'''


def test_no_split_costs_less_and_the_search_is_short(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout

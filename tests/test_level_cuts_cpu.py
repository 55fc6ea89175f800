"""CPU: the search for how a launch over the levels of a pyramid is cut (kernels.h, cheapest_cut) finds what trying every cut finds."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

HARNESS = r"""
#include <cstdio>
#include <random>
#include "kernels.h"
using namespace sfb;

int main() {
  std::mt19937 rng(7);
  auto pick = [&](int lo, int hi) { return (int)std::uniform_int_distribution<int>(lo, hi)(rng); };
  int searched = 0, cut = 0;
  for (int run = 0; run < 20000; ++run) {
    const int levels = pick(1, 4), most0 = pick(1, MAX_PIECES), most1 = pick(1, MAX_PIECES);
    int tiles[4], length[4];
    for (int l = 0; l < levels; ++l) { tiles[l] = pick(0, 1 << pick(0, 9)); length[l] = pick(1, 1 << pick(0, 10)); }
    const double start = pick(0, 10), fold = pick(0, 6);
    const bool both = pick(0, 1) != 0;
    int tried = 0;
    auto fill = [&](auto& work, int n0, int n1) {
      for (int l = 0; l < levels; ++l) {
        const int n = l == 0 || both ? n0 : (l == 1 ? n1 : 1), per = length[l] / n, extra = length[l] - per * n;
        if (run % 2) {
          work.add(tiles[l] * n, (double)length[l] / n + start);
        } else {
          work.add(tiles[l] * extra, per + 1 + start);
          work.add(tiles[l] * (n - extra), per + start);
        }
      }
      return n0 > 1 || n1 > 1 ? fold : 0.0;
    };
    int b0 = 1, b1 = 1;
    double best = 0;
    for (int n0 = 1; n0 <= most0; ++n0)
      for (int n1 = 1; n1 <= std::min(n0, most1); ++n1) {
        BlockQueue queue;
        BlockWork work;
        const double beside = fill(queue, n0, n1), cost = queue.makespan() + beside;
        fill(work, n0, n1);
        if (work.bound() > queue.makespan() * (1 + 1e-9)) { std::printf("bound %g above makespan %g\n", work.bound(), queue.makespan()); return 1; }
        if (best == 0 || cost < 0.95 * best) { best = cost; b0 = n0; b1 = n1; }
        ++tried;
      }
    const LevelCut c = cheapest_cut(most0, most1, fill);
    if (c.n0 != b0 || c.n1 != b1) { std::printf("run %d: %d %d instead of %d %d\n", run, c.n0, c.n1, b0, b1); return 1; }
    searched += tried;
    cut += b0 > 1;
  }
  std::printf("%d cuts, %d launches cut\n", searched, cut);
  return cut > 1000 ? 0 : 2;
}
"""


def test_same_cut_as_trying_all(tmp_path):
    if shutil.which("g++") is None or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("needs g++ and the CUDA headers")
    src = tmp_path / "cuts.cpp"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(CUDA, "include"), "-I", os.path.join(ROOT, "separableflowthesis_b200", "csrc"), "-o",
                    str(tmp_path / "cuts"), str(src)], check=True)
    res = subprocess.run([str(tmp_path / "cuts")], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout

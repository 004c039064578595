"""The row-wise plane-wave basis (basis.cpp) against a scan of the whole box
with the same expression per point: the same points in the same order, over
skewed cells, odd and even boxes, cutoffs that leave rows empty or fill the
box, and k points far outside the first zone, where the basis is empty."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "deepaw-half_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <random>
#include "context.h"

using namespace hb;

int main() {
  std::mt19937 gen(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  long long points = 0;
  for (int t = 0; t < 400; ++t) {
    Crystal c;
    for (int i = 0; i < 9; ++i) c.lattice[i] = (i % 4 == 0 ? 4.0 : 0.0) + (t % 3 ? 2.0 : 0.0) * u(gen);
    if (t % 50 == 7)   // a needle: one long axis
      for (int j = 6; j < 9; ++j) c.lattice[j] *= 40.0;
    const std::array<int, 3> shape = {8 + t % 7, 9 + t % 5, 10 + t % 11};
    const double encut = t % 10 == 3 ? 1e4 : 20.0 + 200.0 * (u(gen) + 1.0);
    double k[3] = {u(gen), u(gen), u(gen)};
    const double far[8] = {-1e10, 1e10, -3e9, 3e9, -2147483648.5, 1e300, -1e300, 12.0};
    if (t % 4 == 0) k[t / 4 % 3] = far[t / 12 % 8];
    const Basis b = build_basis(c, shape, encut, k);
    const auto rec = c.reciprocal();
    size_t at = 0;
    for (int n1 = -(shape[0] / 2); n1 <= (shape[0] - 1) / 2; ++n1)
      for (int n2 = -(shape[1] / 2); n2 <= (shape[1] - 1) / 2; ++n2)
        for (int n3 = -(shape[2] / 2); n3 <= (shape[2] - 1) / 2; ++n3) {
          double q[3];
          for (int j = 0; j < 3; ++j)
            q[j] = (n1 + k[0]) * rec[j] + (n2 + k[1]) * rec[3 + j] + (n3 + k[2]) * rec[6 + j];
          if (!(kHsqdtm * (q[0] * q[0] + q[1] * q[1] + q[2] * q[2]) < encut)) continue;
          if (at >= size_t(b.npw()) || b.gvec[3 * at] != n1 || b.gvec[3 * at + 1] != n2 || b.gvec[3 * at + 2] != n3) {
            std::printf("case %d: point %zu (%d %d %d) differs\n", t, at, n1, n2, n3);
            return 1;
          }
          ++at;
        }
    if (at != size_t(b.npw())) { std::printf("case %d: %zu points, basis has %lld\n", t, at, (long long)b.npw()); return 2; }
    points += (long long)at;
  }
  std::printf("%lld points\n", points);
  return points > 10000 ? 0 : 3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_rows_match_the_whole_box(tmp_path):
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or
                                                                        "/usr/local/cuda/bin/nvcc"))), "include")
    src, exe = tmp_path / "basis.cpp", tmp_path / "basis"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I" + CSRC, "-I" + cuda,
                    "-I" + os.path.join(ROOT, "include"), str(src), os.path.join(CSRC, "basis.cpp"),
                    os.path.join(CSRC, "io.cpp"), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout

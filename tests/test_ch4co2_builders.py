"""Host builders of the CH4-CO2 dipole tables, which every process that binds the system runs:
the coupled form is a small part of their time (a third before its ladder of slices touched
only the slices), and its 591 cubics in 156 groups are the ones the kernel is sized for.  The
fastest of three runs of each, compared within one process."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hawaiihybrid_b200", "csrc")
SRC = r"""
#include <chrono>
#include <cmath>
#include <cstdio>
#include <vector>
#include "hh_ch4co2_coupled.h"
#include "hh_ch4co2_fold.h"
int main() {
  using clk = std::chrono::steady_clock;
  double best[2] = {1e9, 1e9}, sum = 0.0;
  int bad = 0, n_coef = 0, n_group = 0;
  for (int i = 0; i < 3; ++i) {
    const auto a = clk::now();
    Ch4Co2FoldHost f;
    std::vector<float> blob;
    bad |= ch4co2_build_fold(&f) | ch4co2_build_tc_blob(f, &blob);
    const auto b = clk::now();
    Ch4Co2CoupledHost c;
    bad |= ch4co2_build_coupled(&c);
    const auto d = clk::now();
    best[0] = std::fmin(best[0], std::chrono::duration<double>(b - a).count());
    best[1] = std::fmin(best[1], std::chrono::duration<double>(d - b).count());
    n_coef = c.n_coef;
    n_group = c.n_group;
    sum = 0.0;
    for (double x : c.coef) sum += std::fabs(x);
  }
  std::printf("%d %d %d %.17g %.9f %.9f\n", bad, n_coef, n_group, sum, best[0], best[1]);
}
"""


def test_coupled_builder(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-I", CSRC, "-o", exe, str(tmp_path / "t.cpp"),
                    os.path.join(CSRC, "hh_ch4co2_host.cpp")], check=True)
    bad, n_coef, n_group, s, others, coupled = subprocess.run([exe], check=True, capture_output=True,
                                                              text=True).stdout.split()
    assert int(bad) == 0 and (int(n_coef), int(n_group)) == (591, 156)
    assert float(s) > 0.0
    assert float(coupled) < 0.15 * float(others), (coupled, others)

"""How cross-validation groups its folds (csrc/cv_batches.hpp, compiled and run
on the host): the CTA share never looks at free memory, and free memory is asked
for only where the folds are not small beside the device."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fastpls_b200", "csrc")

PROGRAM = r"""
#include "cv_batches.hpp"
#include <cstdio>

int main() {
  const double device = 180e9;
  const int cap = 296;
  for (int folds : {1, 2, 3, 5, 10, 37, 400})
    for (double fold : {65e6, 70e6, 200e6, 900e6, 5e9, 20e9})
      for (int need : {1, 4, 25, 50, 74, 184, 296})
        for (bool alone : {false, true}) {
          auto ctas = [&](int share) { return share > 0 && share < need ? share : need; };
          fpls::CvBatches roomy;
          for (double free : {0.9, 0.3, 0.05, 0.008, 0.0001}) {
            int asked = 0;
            const auto b = fpls::cv_batches(folds, fold, device, cap, alone, ctas, [&] {
              ++asked;
              return free * device;
            });
            if (free == 0.9) roomy = b;
            if (b.max_ctas != roomy.max_ctas) return 1;              // the share followed free memory
            if (b.per_batch < 1 || b.per_batch > roomy.per_batch) return 2;
            if (b.per_batch > 1 && b.per_batch * ctas(b.max_ctas) > cap) return 3;
            if (alone && b.per_batch != 1) return 4;
            if (roomy.per_batch * fold <= device / 32 ? asked : !asked) return 5;
            if (asked && b.per_batch > 1 && b.per_batch * fold > 0.25 * free * device) return 6;
          }
        }
  // lanes only where the component loops are chains of kernels
  if (fpls::fold_lanes(60, false) != 0 || fpls::fold_lanes(2, true) != 2 || fpls::fold_lanes(60, true) != fpls::kLanes)
    return 9;
  // a method without persistent fits, and a device without cooperative launches
  const auto none = [] { return 1e12; };
  const auto all = [](int) { return 296; };
  if (fpls::cv_batches(10, 70e6, device, -1, false, all, none).per_batch != 10) return 7;
  const auto b = fpls::cv_batches(10, 70e6, device, 0, false, all, none);
  return b.per_batch == 1 && b.max_ctas == 0 ? 0 : 8;
}
"""


def test_grouping(tmp_path):
    src = tmp_path / "batches.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "batches"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0

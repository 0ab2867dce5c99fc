"""The order in which the solute sweep's units are handed out
(fx_unit_order.h): every unit of steps x strips once, and behind the three
units it waits for, whatever the two counts, so that a kernel that hands them
out in this order cannot wait for a unit that nobody has taken."""
import os
import subprocess

import conftest

SRC = r"""
#include "fx_unit_order.h"
#include <vector>
int main() {
  for (int steps = 1; steps <= 66; ++steps)
    for (int strips = 1; strips <= 150; ++strips) {
      std::vector<int> at(steps * strips, -1);
      fx_unit_walk w{0, 0};
      for (int i = 0; i < steps * strips; ++i) {
        int jj, s;
        fx_unit_at(i, steps, strips, w, jj, s);
        if (jj < 0 || jj >= steps || s < 0 || s >= strips || at[jj * strips + s] >= 0) return 1;
        at[jj * strips + s] = i;
        if (s > 0 && at[jj * strips + s - 1] < 0) return 2;
        if (jj > 0 && at[(jj - 1) * strips + s] < 0) return 3;
        if (jj > 0 && s + 1 < strips && at[(jj - 1) * strips + s + 1] < 0) return 4;
      }
    }
  return 0;
}
"""


def test_every_unit_once_and_behind_what_it_waits_for(tmp_path):
    src = tmp_path / "order.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "order")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(conftest.ROOT, "fluxos_cpp_b200", "csrc"),
                    "-o", exe, str(src)], check=True)
    assert subprocess.run([exe]).returncode == 0

"""The synthesis beta pass copies its table rows in whole groups: no (m, n) run
of any bandlimit, real or complex, may reach past the rows that are allocated.
The library's own header gives the rows copied and the rows allocated; the runs
are laid out here (rows ordered by m, then n, then l)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), '..', 'hybridpendulum-up_b200', 'csrc')

PROGRAM = r'''
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include "row_groups.hpp"
int main() {
  for (int B = 2; B <= 32; ++B)
    for (int lo : {0, 1 - B}) {
      long nrows = 0, reach = 0;
      for (int m = lo; m < B; ++m)
        for (int n = 1 - B; n < B; ++n) {
          const int len = B - std::max(std::abs(m), std::abs(n));
          reach = std::max(reach, nrows + rows_copied(len));
          nrows += len;
        }
      if (reach > nrows + kRowPad || rows_copied(B) < B) {
        std::printf("B = %d, m from %d: reads %ld rows of %ld + %d\n", B, lo, reach, nrows, kRowPad);
        return 1;
      }
    }
  return 0;
}
'''


def test_runs_stay_within_the_table(tmp_path):
    cxx = shutil.which('g++')
    if cxx is None:
        pytest.skip('no host compiler')
    src = tmp_path / 'runs.cpp'
    src.write_text(PROGRAM)
    exe = str(tmp_path / 'runs')
    subprocess.run([cxx, '-std=c++17', '-I', CSRC, str(src), '-o', exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

"""The tile search of the columns kernel, compiled from the library's own header and enumerated on the CPU: every tile fits its pitch, its
accumulators and a box of 256 rows, for filters of any reach (a dilation of 128 makes a 3-row filter reach 256 rows)."""
import subprocess

from theano_b200 import build

PROGRAM = r"""
#include <stdio.h>
#include "geometry.h"
using namespace b200;
int main() {
  long long found = 0, wrong = 0, far = 0;
  for (int Eh = 0; Eh <= 600; Eh = Eh < 300 ? Eh + 1 : Eh + 50)
    for (int Ew = 0; Ew < 40; ++Ew)
      for (int Wt : {1, 2, 7, 14, 31, 33, 224})
        for (int Ht : {1, 2, 5, 28, 300})
          for (int n_cols : {32, 96, 192})
            for (int even : {1, 2})
              for (int most = 1; most <= (4 * n_cols <= 512 ? 2 : 1); ++most) {
                const ColsTile t = cols_tile(Wt, Ht, Eh, Ew, n_cols, most, even);
                if (!t.found) { far += Eh >= 256; continue; }
                ++found;
                wrong += t.wt < 1 || t.th < 1 || t.wt % even || t.th % even || t.wt + Ew > t.pitch || t.th + Eh > 256 ||
                         t.th * t.pitch > 128 * t.n_acc || t.n_acc < 1 || t.n_acc > most;
              }
  printf("%lld %lld %lld\n", found, wrong, far);
  return 0;
}
"""


def test_tiles_fit_whatever_the_reach_of_the_filter(tmp_path):
    src, exe = tmp_path / "tile.cpp", tmp_path / "tile"
    src.write_text(PROGRAM)
    # without optimisation a division by zero ends the program, wherever its quotient goes
    subprocess.check_call(["g++", "-O0", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I", build.CSRC, str(src), "-o", str(exe)])
    found, wrong, far = map(int, subprocess.check_output([str(exe)]).split())
    assert found > 100000 and wrong == 0 and far > 10000

"""What a kernel with a ring of asynchronously loaded stages waits for when it gives
up (csrc/ring.h): played through on the CPU, every load that is still on its way is
waited for, and each wait is for the newest stage of its slot, the phase that the
slot's barrier is in."""
import subprocess

from op2b import build as B

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "ring.h"
int main() {
  srand(1);
  for (int trial = 0; trial < 200000; trial++) {
    const int ring = 2 + rand() % 3, turns = 1 + rand() % (ring < 3 ? ring : 3);
    const int total = rand() % 40, steps = rand() % 120;
    std::vector<int> last(turns), begun(total, 0), landed(total, 0);
    for (int w = 0; w < turns; w++) last[w] = w - turns;
    int used = 0;  // stages used, in order
    for (int i = 0; i < steps; i++) {
      const int what = rand() % 3, w = rand() % turns;
      if (what == 0) {  // warp w begins its next stage if the slot's last use is over
        const int n = last[w] + turns;
        if (n < total && n - ring < used) begun[n] = 1, last[w] = n;
      } else if (what == 1) {  // a load lands
        const int n = total ? rand() % total : 0;
        if (total && begun[n]) landed[n] = 1;
      } else if (used < total && landed[used]) {
        used++;
      }
    }
    for (int s = 0; s < ring; s++) {
      const int n = op2b::newest_in_flight(s, ring, last.data(), turns);
      int newest = -1;
      for (int m = s; m < total; m += ring)
        if (begun[m]) newest = m;
      for (int m = s; m < total; m += ring)
        if (begun[m] && !landed[m] && m != n) return printf("stage %d not waited for\n", m), 1;
      if (n >= 0 && n != newest) return printf("stage %d is not slot %d's newest\n", n, s), 1;
    }
  }
  return 0;
}
"""


def test_every_load_in_flight_is_waited_for(tmp_path):
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + B.CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout

"""dv_tiles.h: the tiles of a scene are dealt to its team once each, and the walk
over all tiles meets a member's contact tiles in the order of the walk over the
contact tiles alone, in every launch shape, with bilateral rows and without."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <stdio.h>
#include <vector>
#include "dv_tiles.h"
int main() {
  long bad = 0;
  for (int contiguous = 0; contiguous < 2; ++contiguous)
    for (int chunk : {1, 2, 4})
      for (int m : {1, 2, 3, 5, 8, 296})
        for (int ntc = 0; ntc < 40; ++ntc)
          for (int rows : {0, 1, 2, 7}) {
            const int nt = ntc + rows;
            std::vector<int> seen(nt, 0);
            for (int r = 0; r < m; ++r) {
              const dv::TileShare t{r, m, chunk, contiguous};
              std::vector<int> all, contacts;
              for (int i = 0; i < 2 * nt + 8; ++i) {
                const int x = dv::scene_tile(t, ntc, nt, i);
                if (x < 0) break;
                if (x >= nt) return 2;
                ++seen[x];
                if (x < ntc) all.push_back(x);
              }
              for (int i = 0; i < 2 * nt + 8; ++i) {
                const int x = dv::share_tile(t, ntc, i);
                if (x < 0) break;
                contacts.push_back(x);
              }
              bad += all != contacts;
            }
            for (int n : seen) bad += n != 1;
          }
  printf("%ld\n", bad);
  return bad != 0;
}
"""


def test_both_walks_meet_the_same_contact_tiles(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I",
                           os.path.join(ROOT, "dvide_b200", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout

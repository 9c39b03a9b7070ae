"""The columns that a lane of the few-row GEMM reads of the rows it normalises, walked on the host over every row length."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pega_omni_b200" / "csrc"

WALK = r"""
#include <cstdio>
#include <vector>
#include "few_share.h"
using namespace omni;
int main() {
  for (int K = 64; K <= 4096; K += 64)
    for (int rows = 1; rows <= 8; ++rows) {
      const int nkb = K / 64, span = few_span(nkb, 1), per = few_per(nkb, 1), log2 = few_lanes_log2(rows);
      std::vector<int> seen(rows * K / 8, 0);
      for (int warp = 0; warp < kFewWarps; ++warp)
        for (int lane = 0; lane < 32; ++lane) {
          const int kb0 = few_first(warp, 0, span, per), nk = few_count(warp, 0, span, per, nkb);
          const FewShare h = few_share(lane, kb0, nk, log2, rows);
          const int rounds = (per * 8 + h.lanes - 1) / h.lanes;
          for (int j = 0; j < rounds; ++j) {
            const long long at = few_at(h, K) + few_step(h, j);
            if (at < 0 || at % 8 || at + 8 > (long long)rows * K) {
              printf("K %d rows %d warp %d lane %d piece %d: element %lld\n", K, rows, warp, lane, j, at);
              return 1;
            }
            if (h.live && h.first + j * h.lanes < h.pieces) ++seen[at / 8];
          }
        }
      for (int i = 0; i < rows * K / 8; ++i)
        if (seen[i] != 1) {
          printf("K %d rows %d: piece %d is taken %d times\n", K, rows, i, seen[i]);
          return 1;
        }
    }
  return 0;
}
"""


def test_every_piece_is_read_once_and_nothing_outside(tmp_path):
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(WALK)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout

"""Rounds of the dataflow gathers: every position once, no shift beyond the mask.

A thread of a gather marks its missing positions in 32 bits and looks at U of
them at a time (3 and 6 in FP64, 4 and 8 in FP32).  The loop of flow_gather in
solve.cu is replayed here over the shares that the header gives it, for the
gathers of up to three rounds that fronts of thousands of rows make.
"""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "orbit_b200", "csrc")

REPLAY = r"""
#include <cstdio>
#include <vector>
#include "symbolic.h"
using namespace orbit;
int main() {
  const int nt = 128, us[] = {3, 4, 6, 8};
  for (int U : us)
    for (int cnt = 0; cnt <= 10000; cnt += cnt % 1000 < 40 || (cnt > 3800 && cnt < 4150) ? 1 : 37) {
      const int window = flow_window(U);
      std::vector<char> seen(cnt, 0);
      for (int base = 0; base < cnt; base += window * nt)
        for (int tid = 0; tid < nt; ++tid) {
          const FlowShare sh = flow_share(cnt, base, tid, nt, window);
          const unsigned todo = sh.mine == 32 ? 0xffffffffu : (1u << sh.mine) - 1u;
          if (sh.mine > 32 || sh.mine > sh.most) return std::printf("share %d %d %d\n", U, cnt, tid), 1;
          for (int j = 0; j < sh.most; j += U)
            for (int u = 0; u < U; ++u) {
              if (j + u >= 32) return std::printf("U %d, %d positions: shift by %d\n", U, cnt, j + u), 1;
              if (!((todo >> (j + u)) & 1u)) continue;
              const int q = base + (j + u) * nt + tid;
              if (q >= cnt || seen[q]++) return std::printf("U %d, %d positions: position %d\n", U, cnt, q), 1;
            }
        }
      for (char c : seen)
        if (!c) return std::printf("U %d, %d positions: one is left out\n", U, cnt), 1;
    }
  return 0;
}
"""


def test_rounds_cover_every_position_within_the_mask(tmp_path):
    src, exe = tmp_path / "replay.cpp", tmp_path / "replay"
    src.write_text(REPLAY)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

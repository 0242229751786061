"""The launch grids (frg_kernels.h) over SM counts, path counts and every blocks_per_sm that a
configuration may hold, up to the largest int: blocks and warps stay in their ranges, a
larger blocks_per_sm never means fewer of either, and the launch holds the paths that it can."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "finite_root_generation_gb300", "csrc")

MAIN = r"""
#include <limits.h>
#include "frg_kernels.h"
int main() {
  int bad = 0;
  for (int sms : {1, 2, 148, 152})
    for (int64_t n : {(int64_t)1, (int64_t)3, (int64_t)150, (int64_t)607, (int64_t)2049, (int64_t)65536, (int64_t)1 << 33}) {
      for (bool lo : {false, true}) {
        TeamGrid last{0, 0};
        for (int bps : {1, 2, 3, 4, 5, 64, 1 << 20, 600000000, 1073741825, INT_MAX}) {
          const TeamGrid g = frg_team_grid(sms, bps, n, lo);
          const int64_t held = (int64_t)g.blocks * g.warps, before = (int64_t)last.blocks * last.warps;
          const int64_t room = (int64_t)sms * ((int64_t)bps * 4 / g.warps) * g.warps;  // paths that may be resident
          const bool ok = g.blocks >= 1 && g.warps >= 4 && g.warps <= (lo ? 16 : 4) && g.warps % 4 == 0 && held >= before &&
                          (held >= (n < room ? n : room) || g.blocks == INT_MAX);
          if (!ok) { printf("team: %d SMs, %lld paths, %d per SM: %d x %d\n", sms, (long long)n, bps, g.blocks, g.warps); ++bad; }
          last = g;
        }
      }
      int last = 0;
      for (int bps : {1, 2, 3, 64, 1 << 20, 14126300, 600000000, INT_MAX}) {
        const int g = frg_warp_grid(sms, bps, n), t = frg_thread_grid(sms, bps, n);
        const int64_t want = (n + 3) / 4;
        if (g < last || g < 1 || g > want || t < 1 || (bps == INT_MAX && g < want && g < INT_MAX)) {
          printf("warp: %d SMs, %lld paths, %d per SM: %d\n", sms, (long long)n, bps, g);
          ++bad;
        }
        last = g;
      }
    }
  return bad != 0;
}
"""


def test_grids(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-w", f"-I{os.path.join(HERE, 'warp_emu')}", f"-I{CSRC}",
                    str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr

"""Tile geometry of the FP64 grouped kernel (tile_step, warp_grid in
csrc/tsc_kernels.cuh), compiled for the host: every group size is covered by its
tiles exactly once, no tile is empty or larger than its limit, and the four warps
of a tile cover its sub-tiles within what one warp can hold."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "tsc_kernels.cuh"
#include <cstdio>
int main() {
  for (int tile : {32, 48, 64})
    for (int n = 1; n <= 3000; ++n) {
      const int tiles = (n + tile - 1) / tile, step = tsc::tile_step(n, tile);
      if (step > tile || step % 8 || (tiles - 1) * step >= n || tiles * step < n) return std::printf("step %d %d\n", tile, n), 1;
    }
  const int lim[2][2] = {{4, 3}, {2, 2}};
  for (auto& l : lim)
    for (int m = 1; m <= 2 * l[0]; ++m)
      for (int n = 1; n <= 2 * l[1]; ++n) {
        int wm, wn;
        tsc::warp_grid(m, n, l[0], l[1], wm, wn);
        const int mh = (m + wm - 1) / wm, nh = (n + wn - 1) / wn;
        if (wm * wn != 4 || mh > l[0] || nh > l[1] || mh * wm < m || nh * wn < n) return std::printf("warps %d %d\n", m, n), 1;
      }
  std::puts("ok");
}
"""


def test_tiles_cover_groups_and_warps_cover_tiles(tmp_path):
    src = tmp_path / "geom.cpp"
    src.write_text(SRC)
    exe = tmp_path / "geom"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "tsc_tri_t1t2j1j2_b200", "csrc"),
                    "-I", os.path.join(cuda, "include"), "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "ok"

"""Tile shapes of the level-1 operators (ku_shape, filter_shape) on the host: every grid gets one, tiles and chunks cover
it, and a tile fits its CTA.  Sizes from the smallest grid to one of more than 2^29 nodes (fields of more than 4 GB)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "top3d_xl_b200")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

PROGRAM = r"""
#include <cstdio>
#include "topx_opt.cuh"
template <typename S>
bool good(const S& s, const topx::Grid& g, int rows, int even) {
  return s.TY % even == 0 && s.PY == s.TY + 2 && s.PX == s.TX + 2 && s.PY * s.PX <= 256 && s.zc >= 1 &&
         int64_t(s.grid.x) * s.TY >= rows && int64_t(s.grid.y) * s.TX >= g.nnx() && int64_t(s.grid.z) * s.zc >= g.nnz() &&
         s.grid.y < 65536 && s.grid.z < 65536;
}
int main() {
  const int sizes[][3] = {{8, 8, 8}, {8, 16, 1024}, {16, 32, 16}, {24, 1024, 8}, {1024, 8, 8}, {128, 256, 128}, {192, 384, 192},
                          {400, 800, 400}, {816, 808, 816}, {1024, 1024, 640}};
  int bad = 0;
  for (auto& n : sizes) {
    topx::Grid g;
    const int rows = n[0] + 1;
    g.ny = (rows + 3) / 4 * 4 - 1;
    g.nx = n[1];
    g.nz = n[2];
    g.stride = (g.nnodes() + 31) / 32 * 32;
    try {
      if (!good(topx::ku_shape(g, rows), g, rows, 2)) ++bad, std::printf("ku %d %d %d\n", n[0], n[1], n[2]);
      if (!good(topx::filter_shape(g, rows, 8), g, rows, 2)) ++bad, std::printf("filter %d %d %d\n", n[0], n[1], n[2]);
      if (!good(topx::filter_shape(g, rows, 4), g, rows, 4)) ++bad, std::printf("filter32 %d %d %d\n", n[0], n[1], n[2]);
    } catch (const std::exception& e) {
      ++bad;
      std::printf("%d %d %d: %s\n", n[0], n[1], n[2], e.what());
    }
  }
  return bad != 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_every_grid_has_a_tile(tmp_path):
    lib = os.path.join(PKG, "libtopx.so")
    if not os.path.exists(lib):
        pytest.skip("libtopx.so is not built")
    src, exe = tmp_path / "shapes.cu", tmp_path / "shapes"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(PKG, "csrc"), str(src), lib, "-Xlinker", "-rpath", "-Xlinker", PKG, "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

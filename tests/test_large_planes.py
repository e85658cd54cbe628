"""Offsets in planes of more than 2^31 (and, in FP32, 2^32) cells.  Such a grid
takes 50 to 180 GB on the device, so the offsets are computed on the CPU by the
functions that the kernels call, for the cells of the first, the last and the
middle tiles' frames and neighbourhoods."""
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "eshwar_dipan_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "gp_smooth.cuh"
using namespace gpd;
static long long bad = 0, seen = 0;
static void expect(bool ok) { seen++; bad += !ok; }
template <typename R>
static void grid(int mx, int my, int bc) {
  Grid g = {};
  g.mx = mx; g.my = my; g.pitch = (my + 31) / 32 * 32; g.plane = (long long)g.pitch * mx;
  Consts<R> D = {};
  for (int f = 0; f < 2; f++)
    for (int k = 0; k < 2; k++) D.bc_x[f][k] = D.bc_y[f][k] = bc;
  const int xs[3] = {0, mx / 2, mx - TX}, ys[3] = {0, my / 2, my - TY};
  for (int x0 : xs)
    for (int y0 : ys)
      for (int i = -2; i < TX + 2; i++)
        for (int j = -2; j < TY + 2; j++) {
          const int x = x0 + i, y = y0 + j;
          if (x < -2 || x > mx + 1 || y < -2 || y > my + 1) continue;
          const int r = remap(x, mx, bc, bc), c = remap(y, my, bc, bc);
          const __int128 ref = (__int128)r * g.pitch + c;
          const long long o = plane_offset(g, r, c);
          expect((__int128)o == ref && o >= 0 && o < g.plane);
          if (x < 0 || x >= mx || y < 0 || y >= my) continue;
          const auto n = nbr3<R>(D, g, 0, x, y);
          for (int u = 0; u < 3; u++)
            for (int v = 0; v < 3; v++)
              expect((__int128)n.o(u, v) ==
                     (__int128)remap(x - 1 + u, mx, bc, bc) * g.pitch + remap(y - 1 + v, my, bc, bc));
        }
}
int main() {
  for (int bc : {GP_BC_NEUMANN, GP_BC_PERIODIC}) {
    grid<double>(46400, 46400, bc);     /* 2.15e9 cells */
    grid<double>(60000, 62000, bc);     /* 3.72e9 cells */
    grid<double>(262136, 8200, bc);
    grid<float>(46400, 46400, bc);
    grid<float>(80000, 90000, bc);      /* 7.2e9 cells */
    grid<float>(3400, 2000000, bc);
  }
  printf("%lld of %lld\n", bad, seen);
  return bad != 0;
}
"""


def test_offsets(tmp_path):
    sys.path.insert(0, ROOT)
    from eshwar_dipan_b200.build import ARCH, INC, NVCC
    src = tmp_path / "offsets.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "offsets")
    r = subprocess.run([NVCC, *ARCH, "-std=c++17", *INC, str(src), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    bad, seen = re.match(r"(\d+) of (\d+)", r.stdout).groups()
    assert int(seen) > 10000 and int(bad) == 0 and r.returncode == 0, r.stdout


def test_frame_staging_uses_them():
    with open(os.path.join(CSRC, "gp_fused.cuh")) as f:
        src = f.read()
    a = src.index("rows and columns of the frame after the boundary remap")
    body = src[a:src.index("fence_proxy_async_smem();", a)]
    assert "pitch" not in body and body.count("plane_offset(g, ") == 2

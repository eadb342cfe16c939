"""CPU: the cut of a grid into on-chip tiles (csrc/tile_plan.h) against an exhaustive
search of every band's depth: whatever fits in so many tiles is found, the tiles cover
the grid, and each is within its limits."""
import subprocess

import pytest

from seidart_gb300 import build

PROGRAM = r"""
#include <cstdio>
#include "tile_plan.h"
using namespace sfd;

int main() {
  unsigned seed = 1;
  auto rnd = [&](int lo, int hi) { seed = seed * 1664525u + 1013904223u; return lo + (int)((seed >> 8) % (unsigned)(hi - lo + 1)); };
  int fitting = 0, bad = 0;
  for (int n = 0; n < 6000; ++n) {
    const int cells = n % 2 ? 2 : 4, cols = 32 * cells, words = n % 2 ? 12 : 4;
    const TileRules t{cells, 4, n % 2 ? 3 : 4, 16, 0.7, 0.5, 16.0};
    const int W = rnd(1, 20), NX = rnd(2 * W + 4, 1500), NZ = rnd(2 * W + 4, 1500), ctas = rnd(20, 152);
    const size_t limit = 224256;
    auto smem = [&](const Frame& f, int rb) {  // coefficients, halo and its lists, strips: the runs' own sizes
      const size_t R = (size_t)(f.rows + rb - 1) / rb * rb, h = f.rows - f.own;
      return 4 * (size_t)(24 * cols + words * cols * R + (words + 2) * (h * cols + 8 * f.own) + 4 * h * cols +
                          2 * cols * (f.zlo + f.zhi) + 12 * R * f.xlanes);
    };
    TilePlan p{};
    const bool got = plan_tiles(t, NX, NZ, W, ctas, limit, smem, &p);
    // bands of each of the plan's columns, every depth tried, any cost
    const int ng = (NX + cells - 1) / cells, hg = t.halo / cells, inner = 32 - 2 * hg;
    const int ntx = NX <= cols ? 1 : std::max(2, (ng - 2 * hg + inner - 1) / inner);
    int total = 0;
    for (int c = 0; c < ntx && total <= ctas; ++c) {
      auto bound = [&](int q) {
        const int g = ng <= inner * ntx || ntx == 1 ? (int)((long)q * ng / ntx) : q == 0 ? 0 : q == ntx ? ng : inner * q + hg;
        return std::min(NX, cells * g);
      };
      for (int z = 0; z < NZ && total <= ctas; ++total) {
        int z1 = z;
        for (int m = z + 1; m <= std::min(NZ, z + t.max_rb * t.max_warps); ++m) {
          if (m < NZ && NZ - m < t.halo) continue;
          const Frame f = frame_of(NX, NZ, W, cells, t.halo, bound(c), bound(c + 1), z, m);
          if (f.rows <= t.max_rb * t.max_warps && smem(f, t.max_rb) <= limit) z1 = m;
        }
        if (z1 == z) total = ctas + 1;
        z = z1;
      }
    }
    fitting += total <= ctas;
    if (total <= ctas && !got) { ++bad; printf("%d x %d, strips %d, %d tiles: not found\n", NX, NZ, W, ctas); }
    if (!got) continue;
    long covered = 0;
    for (int b = 0; b < p.ntiles; ++b) {
      const int x0 = p.tile[b].x & 0xffff, x1 = p.tile[b].x >> 16, z0 = p.tile[b].y & 0xffff, z1 = p.tile[b].y >> 16;
      const Frame f = frame_of(NX, NZ, W, cells, t.halo, x0, x1, z0, z1);
      covered += (long)(x1 - x0) * (z1 - z0);
      if (x1 <= x0 || z1 <= z0 || f.rows > p.rb * p.warps || smem(f, p.rb) > limit || (z1 < NZ && z1 - z0 < 1)) ++bad;
    }
    if (covered != (long)NX * NZ || p.ntiles > ctas) ++bad;
  }
  printf("%d fit, %d bad\n", fitting, bad);
  return bad != 0 || fitting < 1000;
}
"""


def test_every_grid_that_fits_is_tiled(tmp_path):
    src, exe = tmp_path / "plan.cu", tmp_path / "plan"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc_path(), *build.ARCH, "-std=c++17", "-O1", f"-I{build.CSRC}", f"-I{build.ROOT / 'include'}",
                    "-o", str(exe), str(src)], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:]

// Host side of the on-chip tiles (em2_tile.cuh): a tile's frame and the cut of
// a grid into tiles.
#pragma once
#include <algorithm>
#include <vector>

#include "resident.h"

namespace sfd {

// The frame of a tile of `cells` cells a lane with `halo` cells of halo.
struct Frame {
  int rows, own, zlo, zhi, xlanes;  // rows, owned ones, those of the low and the high z strip, lanes with x-strip cells
  int zhi0;                         // first row of the high z strip, of two rows at least
  bool edge;                        // it holds strip or boundary cells
};

inline Frame frame_of(int NX, int NZ, int W, int cells, int halo, int ox0, int ox1, int oz0, int oz1) {
  const int bx = ox0 > 0 ? ox0 - halo : 0, bz = std::max(oz0 - halo, 0);
  const int xend = std::min(NX, ox1 + halo), kend = std::min(NZ, oz1 + halo);
  Frame f;
  f.rows = kend - bz;
  f.own = oz1 - oz0;
  f.zlo = std::max(std::min(W, kend) - bz, 0);
  f.zhi0 = std::max(NZ - std::max(W, 2), bz) - bz;
  f.zhi = std::max(kend - std::max(NZ - W, bz), 0);
  const int xlo = std::max((std::min(W, xend) - bx + cells - 1) / cells, 0);
  const int xh0 = std::max((NX - W - bx) / cells, xlo);
  f.xlanes = xlo + std::max((xend - bx + cells - 1) / cells - xh0, 0);
  const int lo = std::max(W, 1);
  f.edge = bx < lo || xend > NX - std::max(W, 2) || bz < lo || kend > NZ - std::max(W, 2);
  return f;
}

// What a tiling depends on: cells a lane and of halo, the most rows a warp and
// warps a CTA, and the cost model -- a frame row without strip or boundary
// cells costs 1, one of a z strip zrow more, every row of a tile with strip
// columns xcol of that more; no tile gets less than min_cost.
struct TileRules {
  int cells, halo, max_rb, max_warps;
  double zrow, xcol, min_cost;
};

// Cuts an NX x NZ grid into tile columns -- as few as there can be, of about
// equal width -- and each of them into bands of about equal cost, at most
// max_ctas tiles of smem(frame, rb) <= max_smem bytes.  False when the grid
// does not fit.
template <class Smem>
bool plan_tiles(const TileRules& t, int NX, int NZ, int W, int max_ctas, size_t max_smem, const Smem& smem, TilePlan* out) {
  max_ctas = std::min(max_ctas, kResMaxTiles);
  // column bounds in lanes; an outermost column has one halo less to hold
  const int ng = (NX + t.cells - 1) / t.cells, hg = t.halo / t.cells, inner = 32 - 2 * hg;
  const int ntx = NX <= 32 * t.cells ? 1 : std::max(2, (ng - 2 * hg + inner - 1) / inner);
  if (ntx > max_ctas) return false;
  std::vector<int> xb(ntx + 1);
  for (int c = 0; c <= ntx; ++c) {
    const int g = ng <= inner * ntx || ntx == 1 ? (int)((long)c * ng / ntx) : c == 0 ? 0 : c == ntx ? ng : inner * c + hg;
    xb[c] = std::min(NX, t.cells * g);
  }
  const int max_rows = t.max_rb * t.max_warps;
  auto frame = [&](int c, int z0, int z1) { return frame_of(NX, NZ, W, t.cells, t.halo, xb[c], xb[c + 1], z0, z1); };
  // the bands of column c at cost C a tile, greedily from the top
  auto bands = [&](int c, double C, std::vector<int>* cuts) {
    int n = 0, z = 0;
    if (cuts) cuts->assign(1, 0);
    while (z < NZ) {
      auto fits = [&](int m) {
        const Frame f = frame(c, z, m);
        const double cost = (f.rows + t.zrow * (f.zlo + f.zhi)) * (f.xlanes ? 1.0 + t.xcol : 1.0);
        return cost <= C && f.rows <= max_rows && smem(f, t.max_rb) <= max_smem;
      };
      // the deepest band that fits.  Rows, cost and memory grow with it as long as
      // it has its whole halo below; the last one, whose frame ends with the grid,
      // takes less memory than those that end a few rows higher.  So: the rest of the
      // column, or by bisection a band that leaves the last one no thinner than its
      // neighbours' halo.
      int z1 = NZ;
      if (!fits(NZ)) {
        int over = std::min(std::max(NZ - t.halo, z), z + max_rows) + 1;
        z1 = z;
        while (over - z1 > 1) {
          const int m = (z1 + over) / 2;
          (fits(m) ? z1 : over) = m;
        }
      }
      if (z1 == z) return max_ctas + 1;
      z = z1;
      ++n;
      if (cuts) cuts->push_back(z);
      if (n > max_ctas) break;
    }
    return n;
  };
  auto tiles_at = [&](double C) {
    int total = 0;
    for (int c = 0; c < ntx && total <= max_ctas; ++c) total += bands(c, C, nullptr);
    return total;
  };
  double lo = t.min_cost - 0.5, hi = 3.0 * max_rows;
  if (tiles_at(hi) > max_ctas) return false;
  if (tiles_at(lo) <= max_ctas) hi = lo;
  for (int it = 0; it < 24 && hi - lo > 0.25; ++it) {
    const double mid = 0.5 * (lo + hi);
    (tiles_at(mid) <= max_ctas ? hi : lo) = mid;
  }
  out->ntiles = out->ntz = 0;
  int rows = 0;
  std::vector<int> cuts;
  std::vector<Frame> frames;
  for (int c = 0; c < ntx; ++c) {
    bands(c, hi, &cuts);
    out->ntz = std::max(out->ntz, (int)cuts.size() - 1);
    for (size_t q = 0; q + 1 < cuts.size(); ++q) {
      const Frame f = frame(c, cuts[q], cuts[q + 1]);
      rows = std::max(rows, f.rows);
      frames.push_back(f);
      out->tile[out->ntiles++] =
          make_int4(xb[c] | (xb[c + 1] << 16), cuts[q] | (cuts[q + 1] << 16), f.edge ? (f.xlanes ? 2 : 1) : 0, 0);
    }
  }
  out->rb = 1;
  while (rows > out->rb * t.max_warps) ++out->rb;
  out->warps = (rows + out->rb - 1) / out->rb;
  out->smem = 0;
  for (const Frame& f : frames) out->smem = std::max(out->smem, smem(f, out->rb));
  return out->smem <= max_smem;
}

}  // namespace sfd

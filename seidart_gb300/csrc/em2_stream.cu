// Streaming electromag2 runs: grids too large for the chip (and handles told to
// stay off it) advance kTileHalo steps a launch, every launch reading one copy
// of the state and writing the other; what is left of a run takes single steps
// (fused2d.cu; sfd_api.cu says how many).
//
// The tiles are those of the on-chip run (em2_run.cuh): a CTA loads its frame --
// the owned cells, four cells of halo, coefficients and strips' memory
// variables -- advances it by up to four steps on chip and writes the owned
// cells.  The state and the coefficients then cross device memory once in four
// steps instead of once a step.
//
// What bounds it: 4040 x 3040 cells take 43.9 us a step (280 Gcell-updates/s;
// one launch a step took 104 us, 118 Gcell/s and 74 % of the copy bandwidth).
// A launch moves 0.64 GB counting every frame's halo, 95 us at the copy
// bandwidth, and takes 176 us: the rest is a tile's own chain -- its loads, four
// steps of two barriers, its stores -- of which two CTAs an SM hide each
// other's.  2040 x 1540 cells take 14.7 us a step, 1300 x 900 cells 7.4 us.
// Frames of 64 rows (16 warps, one CTA an SM) compute less twice and run 43.2 /
// 15.6 / 8.2 us; of 24 rows (8 warps of 3) 47.7 / 15.0 / 7.8, of 48 rows (16 of
// 3) 46.0 / 14.9 / 7.2.  Coefficients copied to shared memory asynchronously,
// not through registers, let every row's loads be in flight at once and
// took 64-row frames from 48.1 to 43.2 us.
#include <algorithm>

// Rows a warp and warps of a CTA.
#ifndef SFD_EM2_STREAM_RB
#define SFD_EM2_STREAM_RB 4
#endif
#ifndef SFD_EM2_STREAM_WARPS
#define SFD_EM2_STREAM_WARPS 8
#endif
#define EM2_RUN_WARPS SFD_EM2_STREAM_WARPS
#include "em2_run.cuh"

namespace sfd {

namespace {

constexpr int kRows = SFD_EM2_STREAM_RB, kWarps = SFD_EM2_STREAM_WARPS, kFrame = kRows * kWarps;

// Tiles of uniform size: ntx columns of at most 120 cells (one of up to 128),
// nbz bands of at most kFrame - 2 kTileHalo rows (one of up to kFrame).
__host__ __device__ inline int cut_x(int NX, int c, int ntx) {
  const int x = (int)(4 * ((long)((NX + 3) / 4) * c / ntx));
  return x < NX ? x : NX;
}
__host__ __device__ inline int cut_z(int NZ, int r, int nbz) { return (int)((long)NZ * r / nbz); }

template <int RB>
__global__ void __launch_bounds__(32 * kWarps, 16 / kWarps)
    em2_stream_kernel(const __grid_constant__ Em2Resident a, int ntx, int nbz) {
  __shared__ Em2Tile G;
  const int NX = a.NX, NZ = a.NZ, W = a.W;
  const int c = blockIdx.x % ntx, r = blockIdx.x / ntx;
  const int4 te = make_int4(cut_x(NX, c, ntx), cut_x(NX, c + 1, ntx), cut_z(NZ, r, nbz), cut_z(NZ, r + 1, nbz));
  const int bx = max(te.x - kTileHalo, 0), xend = min(NX, te.y + kTileHalo);
  const int bz = max(te.z - kTileHalo, 0), kend = min(NZ, te.w + kTileHalo);
  const bool xs = bx < max(W, 1) || xend > NX - max(W, 2);
  const bool edge = xs || bx < 1 || xend > NX - 2 || bz < max(W, 1) || kend > NZ - max(W, 2);
  if (!edge) em2_run_tile<RB, kStream, false, false>(a, G, te);
  else if (!xs) em2_run_tile<RB, kStream, true, false>(a, G, te);
  else em2_run_tile<RB, kStream, true, true>(a, G, te);
}

}  // namespace

cudaError_t em2_stream_prepare(int NX, int NZ, int W, StreamPlan* out) {
  const int ng = (NX + 3) / 4;
  out->ntx = NX <= kCols ? 1 : (ng + 29) / 30;
  out->nbz = NZ <= kFrame ? 1 : (NZ + kFrame - 2 * kTileHalo - 1) / (kFrame - 2 * kTileHalo);
  // the most rows in warps with a z-strip row and the most lanes with an
  // x-strip cell of any frame, counted as em2_run_tile does
  int zrows = 0, xlanes = 0;
  for (int r = 0; r < out->nbz; ++r) {
    const int bz = std::max(cut_z(NZ, r, out->nbz) - kTileHalo, 0), kend = std::min(NZ, cut_z(NZ, r + 1, out->nbz) + kTileHalo);
    const int wlo = (std::max(std::min(W, kend) - bz, 0) + kRows - 1) / kRows;
    const int wh0 = std::max((std::max(NZ - std::max(W, 2), bz) - bz) / kRows, wlo);
    zrows = std::max(zrows, kRows * (wlo + std::max((kend - bz + kRows - 1) / kRows - wh0, 0)));
  }
  for (int c = 0; c < out->ntx; ++c) {
    const int bx = std::max(cut_x(NX, c, out->ntx) - kTileHalo, 0), xend = std::min(NX, cut_x(NX, c + 1, out->ntx) + kTileHalo);
    const int xlo = std::max((std::min(W, xend) - bx + 3) / 4, 0), xh0 = std::max((NX - W - bx) / 4, xlo);
    xlanes = std::max(xlanes, xlo + std::max((xend - bx + 3) / 4 - xh0, 0));
  }
  out->smem = sizeof(float) * (kOC + (kRows <= kEm2KeepRows ? 0 : 4 * kCols * kFrame) + 2 * kCols * zrows + 8 * kFrame * xlanes);
  return res_allow_max_smem((const void*)em2_stream_kernel<kRows>);
}

void em2_stream_launch(const Em2Resident& a, const StreamPlan& plan, cudaStream_t s) {
  em2_stream_kernel<kRows><<<plan.ntx * plan.nbz, 32 * kWarps, plan.smem, s>>>(a, plan.ntx, plan.nbz);
}

}  // namespace sfd

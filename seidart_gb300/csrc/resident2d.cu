// SM-resident electromag2 run: every time step of an sfd_run in one
// cooperative launch, with the whole state on chip.
//
// The grid is cut into tiles (TilePlan), one CTA each for the whole run.  A
// tile is the frame of em2_tile.cuh: RB rows of 128 columns a warp, the
// fields in registers, coefficients and CPML memory variables in shared
// memory.  Every kTileHalo steps a tile writes the owned cells its
// neighbours' halos hold to global memory (L2) as 16-byte words {Ex, Ez, Hy,
// tag}, indexed by the cell's place in the grid, and reads its own halo
// cells' words until they carry the tag of this hand-over; the words of strip
// cells' memory variables go the same way.  Two copies, by the parity of the
// tag: a tile writes a word again two hand-overs later, after it has read
// words its neighbours wrote one hand-over later, and they had read the first
// by then.  A thread's poll gives up after limit_ns (%globaltimer) or when
// another tile has given up, records the failure in the control block, and
// the CTA leaves the run at the next barrier; the host reports
// SFD_ERR_TIMEOUT.  The launch is cooperative, so all tiles are co-resident
// and a correct run never reaches the limit.
//
// What bounds it: the chain of a step -- two block barriers, a row of shared
// memory each way, about 60 instructions for each row of four cells -- and,
// every fourth step, the hand-over through L2.  On 1040 x 540 cells a step
// takes 1.83 us (1.3 us of it the step of the largest tiles, the rest a
// hand-over of 2.2 us in four); 120 x 90 cells take 1.2 to 1.3 us.  The form before
// it exchanged one-cell edges twice a step, every cell mask applied in the
// step: 4.24 and 4.3 us.
//
// The per-cell arithmetic is that of the loops of
// legacy/fortran/electromagfdtd.f95:249-321.  Every product and sum names its
// rounding, so that a cell gets the same bits from whichever tile computes it
// (its own or one whose halo it lies in) and whichever form of the kernel, here,
// streamed, one step a launch or batched: a run in pieces, with checkpoints or
// recomputed for the adjoint gives the states of the plain run.
#include <algorithm>

#include "em2_run.cuh"
#include "tile_plan.h"

namespace sfd {

using namespace res;
using namespace tile2;

namespace {

template <int RB, int MODE>
__global__ void __launch_bounds__(32 * kEm2MaxWarps, 1) em2_resident_kernel(const __grid_constant__ Em2Resident a) {
  __shared__ Em2Tile G;
  const int4 t = a.plan.tile[blockIdx.x];
  const int4 te = make_int4(t.x & 0xffff, t.x >> 16, t.y & 0xffff, t.y >> 16);
  if (t.z == 0) em2_run_tile<RB, MODE, false, false>(a, G, te);
  else if (t.z == 1 && te.y + kTileHalo <= a.NX - 2) em2_run_tile<RB, MODE, true, false>(a, G, te);
  else em2_run_tile<RB, MODE, true, true>(a, G, te);
}

const void* em2_kernel(int rb, int mode) {
  static const void* const k[kEm2MaxRows][3] = {
      {(const void*)em2_resident_kernel<1, 0>, (const void*)em2_resident_kernel<1, 1>, (const void*)em2_resident_kernel<1, 2>},
      {(const void*)em2_resident_kernel<2, 0>, (const void*)em2_resident_kernel<2, 1>, (const void*)em2_resident_kernel<2, 2>},
      {(const void*)em2_resident_kernel<3, 0>, (const void*)em2_resident_kernel<3, 1>, (const void*)em2_resident_kernel<3, 2>},
      {(const void*)em2_resident_kernel<4, 0>, (const void*)em2_resident_kernel<4, 1>, (const void*)em2_resident_kernel<4, 2>}};
  return k[rb - 1][mode];
}

// Cost model of the planner: a frame row of a tile without strip or boundary
// cells costs 1; a tile with strip columns, and a row of a z strip, this much
// more (measured cycles a step and row: 46 inside, about 80 with either; on
// 1040 x 540 cells weights of 0.4 to 1 change the step by under 6 %).  Tiles
// get no fewer than kMinCost rows' worth: below that the chain of
// a step, not its rows, sets the time, and more tiles only add hand-overs.
#ifndef SFD_EM2_ZROW_COST
#define SFD_EM2_ZROW_COST 0.7
#endif
#ifndef SFD_EM2_XCOL_COST
#define SFD_EM2_XCOL_COST 0.5
#endif
#ifndef SFD_EM2_MIN_COST
#define SFD_EM2_MIN_COST 16.0
#endif

// Shared memory of a frame with rb rows a warp, as em2_run_tile (em2_run.cuh) lays it out.
size_t em2_tile_smem(const Frame& f, int rb) {
  const size_t R = (size_t)(f.rows + rb - 1) / rb * rb;
  const int hrows = f.rows - f.own;
  const int zn = f.edge ? f.zlo + f.zhi : 0, xl = f.edge ? f.xlanes : 0;
  size_t n = kOC + (rb <= kEm2KeepRows ? 0 : 4 * kCols * R) + 3 * ((size_t)hrows * kCols + 8 * (size_t)f.own) + 1 +
             2 * (size_t)(em2_get_entries(hrows, f.own, zn, xl) + em2_pub_entries(f.own, zn, xl));
  if (f.edge) {
    const size_t wlo = (f.zlo + rb - 1) / rb, wh0 = std::max<size_t>(f.zhi0 / rb, wlo);
    n += 2 * kCols * rb * (wlo + (R / rb > wh0 ? R / rb - wh0 : 0)) + 8 * R * (size_t)f.xlanes;
  }
  return sizeof(float) * n;
}

}  // namespace

bool em2_resident_plan(int NX, int NZ, int npml, int max_ctas, size_t max_smem, TilePlan* out) {
  const TileRules rules{4, kTileHalo, kEm2MaxRows, kEm2MaxWarps, SFD_EM2_ZROW_COST, SFD_EM2_XCOL_COST, SFD_EM2_MIN_COST};
  return plan_tiles(rules, NX, NZ, npml, max_ctas, max_smem, em2_tile_smem, out);
}

cudaError_t em2_resident_prepare(const TilePlan& plan, int* ctas_per_sm) {
  int n = 1 << 30;
  for (int mode = 0; mode < 3; ++mode) {
    const void* fn = em2_kernel(plan.rb, mode);
    cudaError_t e = res_allow_max_smem(fn);
    int q = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, fn, 32 * plan.warps, plan.smem);
    if (e != cudaSuccess) return e;
    n = std::min(n, q);
  }
  *ctas_per_sm = n;
  return cudaSuccess;
}

cudaError_t em2_resident_launch(const Em2Resident& a, cudaStream_t s) {
  void* args[] = {(void*)&a};
  const void* fn = em2_kernel(a.plan.rb, a.dump.base ? 1 : a.ckpt.base ? 2 : 0);
  return cudaLaunchCooperativeKernel(fn, dim3(a.plan.ntiles), dim3(32 * a.plan.warps), args, a.plan.smem, s);
}

}  // namespace sfd

// SM-resident seismic2 run (corrected physics): every time step of an sfd_run
// in one cooperative launch, with the whole state on chip.
//
// The tiles are those of the electromag2 run (em2_tile.cuh, resident2d.cu) for
// the velocity-stress step: a warp holds RB whole rows of 64 columns, two cells
// a lane, the five fields in registers; the twelve coefficients lie in
// registers for RB = 1, else in shared memory, the CPML memory variables of
// strip cells in shared memory.  A half-step needs its neighbours along x from
// the next lanes (six shuffles a row and step) and along z from the next warps
// (vx, vz of a warp's first and last row, szz of its first, sxz of its last
// row through shared memory).  A step moves information by two cells -- the
// stresses read velocities one cell away, the velocities stresses one cell away
// -- so a halo of kS2Halo cells lasts kS2Steps steps; then the tiles hand over
// {vx, vz, sxx, tag} and {szz, sxz, -, tag} of every halo cell, and the strips'
// memory variables, through L2 as the electromag2 run does.
//
// The Fortran's loop bounds (seismicfdtd.f95:247-357) are coefficient values:
// sfd_set_model leaves the stiffness averages zero outside their loop, and
// dt/rho of the outermost cells, where the velocities are Dirichlet planes, is
// taken as zero.  A memory variable outside its loop is left to run in shared
// memory -- it is only ever multiplied by such a zero -- and is not stored.
//
// What bounds it: as there, the chain of a step and the hand-over every
// kS2Steps steps.  On 440 x 240 cells a step takes 2.32 us (3.4 us in the form
// before it, which exchanged one-cell edges twice a step and read every operand
// from shared memory), on 120 x 90 cells 1.85 us.  Halos of 6 and 8 cells (3
// and 4 steps a hand-over) run 2.47 and 2.29 us: what they save in hand-overs
// they compute twice.  Frames of one row a warp (21 warps) run 2.84 us.
//
// Every product and sum names its rounding, so that a cell gets the same bits
// from whichever tile computes it and a run in pieces, or recomputed for the
// adjoint, gives the states of the plain run.
#include <algorithm>

#include "s2_run.cuh"
#include "tile_plan.h"

namespace sfd {

namespace {

template <int RB, bool DUMP>
__global__ void __launch_bounds__(32 * kS2Warps, 1) seis2_resident_kernel(const __grid_constant__ Seis2Resident a) {
  __shared__ S2Tile G;
  const int4 t = a.tiles.tile[blockIdx.x], te = make_int4(t.x & 0xffff, t.x >> 16, t.y & 0xffff, t.y >> 16);
  if (t.z == 0) s2_run_tile<RB, DUMP, false, false>(a, G, te);
  else if (t.z == 1) s2_run_tile<RB, DUMP, true, false>(a, G, te);
  else s2_run_tile<RB, DUMP, true, true>(a, G, te);
}

const void* s2_kernel(int rb, bool dump) {
  static const void* const k[kS2MaxRows][2] = {
      {(const void*)seis2_resident_kernel<1, false>, (const void*)seis2_resident_kernel<1, true>},
      {(const void*)seis2_resident_kernel<2, false>, (const void*)seis2_resident_kernel<2, true>},
      {(const void*)seis2_resident_kernel<3, false>, (const void*)seis2_resident_kernel<3, true>}};
  return k[rb - 1][dump];
}

// Shared memory of a frame with rb rows a warp, as s2_run_tile lays it out.
size_t s2_tile_smem(const Frame& f, int rb) {
  const size_t R = (size_t)(f.rows + rb - 1) / rb * rb;
  const int hrows = f.rows - f.own;
  const int zn = f.edge ? f.zlo + f.zhi : 0, xl = f.edge ? f.xlanes : 0;
  size_t n = kSCo + (rb <= kS2Keep ? 0 : 12 * kSC * R) + 6 * ((size_t)hrows * kSC + 2 * kS2Halo * (size_t)f.own) + 1 +
             2 * (size_t)(s2_get_entries(hrows, f.own, zn, xl) + s2_pub_entries(f.own, zn, xl));
  if (f.edge) {
    const size_t wlo = (f.zlo + rb - 1) / rb, wh0 = std::max<size_t>(f.zhi0 / rb, wlo);
    n += 6 * kSC * rb * (wlo + (R / rb > wh0 ? R / rb - wh0 : 0)) + 12 * R * (size_t)f.xlanes;
  }
  return sizeof(float) * n;
}

// The planner's cost model (tile_plan.h).
#ifndef SFD_S2_ZROW_COST
#define SFD_S2_ZROW_COST 0.7
#endif
#ifndef SFD_S2_XCOL_COST
#define SFD_S2_XCOL_COST 0.5
#endif
#ifndef SFD_S2_MIN_COST
#define SFD_S2_MIN_COST 16.0
#endif

}  // namespace

bool seis2_resident_plan(int NX, int NZ, int npml, int max_ctas, size_t max_smem, TilePlan* out) {
  const TileRules rules{2, kS2Halo, kS2MaxRows, kS2Warps, SFD_S2_ZROW_COST, SFD_S2_XCOL_COST, SFD_S2_MIN_COST};
  return plan_tiles(rules, NX, NZ, npml, max_ctas, max_smem, s2_tile_smem, out);
}

cudaError_t seis2_resident_prepare(const TilePlan& plan, int* ctas_per_sm) {
  int n = 1 << 30;
  for (int dump = 0; dump < 2; ++dump) {
    const void* fn = s2_kernel(plan.rb, dump);
    cudaError_t e = res_allow_max_smem(fn);
    int q = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, fn, 32 * plan.warps, plan.smem);
    if (e != cudaSuccess) return e;
    n = std::min(n, q);
  }
  *ctas_per_sm = n;
  return cudaSuccess;
}

cudaError_t seis2_resident_launch(const Seis2Resident& a, cudaStream_t s) {
  void* args[] = {(void*)&a};
  return cudaLaunchCooperativeKernel(s2_kernel(a.tiles.rb, a.dump.base != nullptr), dim3(a.tiles.ntiles),
                                     dim3(32 * a.tiles.warps), args, a.tiles.smem, s);
}

}  // namespace sfd

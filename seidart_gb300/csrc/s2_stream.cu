// Streaming seismic2 runs (corrected physics): grids too large for the chip (and
// handles told to stay off it) advance kS2Steps steps a launch, every launch
// reading one copy of the state and writing the other, where that is faster than
// single steps (fused2d.cu), which what is left of a run takes too.
//
// The tiles are those of the on-chip run (s2_run.cuh): a CTA loads its frame -- the
// owned cells, kS2Halo cells of halo, coefficients and strips' memory variables
// --, advances it by up to two steps on chip and writes the owned cells.
//
// What bounds it: 2040 x 1540 cells take 71 us a step (44 Gcell-updates/s; one
// launch a step took 84 us), 1200 x 900 cells 30 us (36), 801 x 640 15 us (17).  A
// launch moves 0.36 GB counting every frame's halo, 54 us at the copy bandwidth,
// and takes 142 us: a tile's loads, two steps and stores follow one another, and
// frames of 48 x 64 cells with their coefficients leave an SM room for one.
#include <algorithm>

#include "s2_run.cuh"

namespace sfd {

namespace {

// Tiles of uniform size: ntx columns of at most kSC - 2 kS2Halo cells (one of up
// to kSC), nbz bands of at most kS2Warps RB - 2 kS2Halo rows (one of up to kS2Warps RB).
__host__ __device__ inline int cut_x(int NX, int c, int ntx) {
  const int x = (int)(2 * ((long)((NX + 1) / 2) * c / ntx));
  return x < NX ? x : NX;
}
__host__ __device__ inline int cut_z(int NZ, int r, int nbz) { return (int)((long)NZ * r / nbz); }

template <int RB>
__global__ void __launch_bounds__(32 * kS2Warps, 1)
    s2_stream_kernel(const __grid_constant__ Seis2Resident a, int ntx, int nbz) {
  __shared__ S2Tile G;
  const int NX = a.NX, NZ = a.NZ, W = a.W;
  const int c = blockIdx.x % ntx, r = blockIdx.x / ntx;
  const int4 te = make_int4(cut_x(NX, c, ntx), cut_x(NX, c + 1, ntx), cut_z(NZ, r, nbz), cut_z(NZ, r + 1, nbz));
  const int bx = max(te.x - kS2Halo, 0), xend = min(NX, te.y + kS2Halo);
  const int bz = max(te.z - kS2Halo, 0), kend = min(NZ, te.w + kS2Halo);
  const bool xs = bx < W || xend > NX - W;
  const bool edge = xs || bz < W || kend > NZ - W;  // strips are a cell deep at least: the planes lie in them
  if (!edge) s2_run_tile<RB, kS2Stream, false, false>(a, G, te);
  else if (!xs) s2_run_tile<RB, kS2Stream, true, false>(a, G, te);
  else s2_run_tile<RB, kS2Stream, true, true>(a, G, te);
}

using Kernel = void (*)(Seis2Resident, int, int);
Kernel kernel_of(int rb) { return rb == 3 ? s2_stream_kernel<3> : s2_stream_kernel<2>; }

// Shared memory of the largest tile, as s2_run_tile lays it out.
size_t tile_smem(int NX, int NZ, int W, int rb, int ntx, int nbz) {
  size_t most = 0;
  for (int r = 0; r < nbz; ++r) {
    const int bz = std::max(cut_z(NZ, r, nbz) - kS2Halo, 0), kend = std::min(NZ, cut_z(NZ, r + 1, nbz) + kS2Halo);
    const int R = (kend - bz + rb - 1) / rb * rb;
    const int wlo = (std::max(std::min(W, kend) - bz, 0) + rb - 1) / rb;
    const int wh0 = std::max((std::max(NZ - W, bz) - bz) / rb, wlo);
    const int zrows = rb * (wlo + std::max(R / rb - wh0, 0));
    for (int c = 0; c < ntx; ++c) {
      const int bx = std::max(cut_x(NX, c, ntx) - kS2Halo, 0), xend = std::min(NX, cut_x(NX, c + 1, ntx) + kS2Halo);
      const int xlo = std::max((std::min(W, xend) - bx + 1) / 2, 0), xh0 = std::max((NX - W - bx) / 2, xlo);
      const int xlanes = xlo + std::max((xend - bx + 1) / 2 - xh0, 0);
      most = std::max(most, (size_t)kSCo + 12 * kSC * R + 6 * kSC * zrows + 12 * (size_t)R * xlanes);
    }
  }
  return sizeof(float) * most;
}

}  // namespace

// Tiles are worth it where they fill 0.7 of their waves (one CTA an SM): a launch of
// one wave takes 23 us, of two 32, of three 43, whatever the last one holds, and a
// single-pass step 7 us and 20 for a million cells.  (us a step so and so: 440 x 240
// cells, 0.31 of one wave, 11.5 and 8.2; 635 x 460, 0.86, 11.5 and 12.6; 723 x 549,
// 0.58 of two, 15.9 and 15.3; 1036 x 501, 0.76 of two, 15.7 and 17.7; 897 x 907,
// 0.80 of three, 21.4 and 22.7.)
constexpr double kWorth = 0.7;

cudaError_t seis2_stream_prepare(int NX, int NZ, int W, StreamPlan* out, bool* faster) {
  int dev = 0, optin = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  const size_t limit = (size_t)optin - sizeof(S2Tile) - 256;  // the static shared memory (and block_norm_to_slot's)
  const int ng = (NX + 1) / 2, most = (kSC - 2 * kS2Halo) / 2;
  out->ntx = NX <= kSC ? 1 : (ng + most - 1) / most;
  for (out->rb = 3;; --out->rb) {  // three rows a warp, two where wide strips leave them no room (two always fit)
    const int F = kS2Warps * out->rb;
    out->nbz = NZ <= F ? 1 : (NZ + F - 2 * kS2Halo - 1) / (F - 2 * kS2Halo);
    out->smem = tile_smem(NX, NZ, W, out->rb, out->ntx, out->nbz);
    if (out->smem <= limit || out->rb == 2) break;
  }
  const int waves = (out->ntx * out->nbz + sms - 1) / sms;
  const double wave = (double)sms * (kSC - 2 * kS2Halo) * (kS2Warps * out->rb - 2 * kS2Halo);  // cells
  *faster = (double)NX * NZ > kWorth * waves * wave;
  return res_allow_max_smem((const void*)kernel_of(out->rb));
}

void seis2_stream_launch(const Seis2Resident& a, const StreamPlan& plan, cudaStream_t s) {
  kernel_of(plan.rb)<<<plan.ntx * plan.nbz, 32 * kS2Warps, plan.smem, s>>>(a, plan.ntx, plan.nbz);
}

}  // namespace sfd

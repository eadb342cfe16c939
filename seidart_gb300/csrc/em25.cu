// electromag25 (legacy/fortran/electromagfdtd.f95:619-1092): 2.5-D Yee scheme
// with Ex Ey Ez Hx Hy Hz, twelve CPML memory variables and y-invariant
// permittivity / conductivity.  A thread takes four (x, z) columns, marching along y.
//   half1: Hx (:901-919), Hy (:922-940), Hz (:943-962); block (0,0,0) first
//          records the receivers of the previous step.
//   half2: Ex and Ey (:968-1009), Ez (:1012-1029), source (:1033-1035),
//          Dirichlet faces of E (:1038-1055) and the norm (:1081-1082).
// The H faces (:1057-1078) are zeroed at the end of a Fortran step, after the
// E update has read them; half1 treats the previous H on those faces as zero
// and the finalize kernels zero them in memory at the end of each run.
#include <type_traits>
#include "sfd_solvers.h"
#include "tma.cuh"

namespace sfd {

namespace {

// ---------------------------------------------------------------------------
// TMA-staged y-march.  A block takes 32 x TZ columns (four a thread, 8 x TZ
// threads) and one y segment, and streams the segment's y planes through a ring
// of kRing shared-memory stages filled by cp.async.bulk.tensor boxes that one
// thread issues ahead, completion on the stage's mbarrier:
//   H kernel: the three E fields of the own cells and the next ones up x and z
//             (x from i0, rows k0 .. k0 + TZ) and the three H fields of the own
//             cells; the plane after the segment is staged too (its E only) for
//             the y+ differences;
//   E kernel: the three H fields of the own cells and the ones before down x
//             and z (x from i0 - 4, rows k0 - 1 .. k0 + TZ - 1) and the three E
//             fields of the own cells; the y- values are carried in registers.
// The memory variables (strips only) and the results go through plain 16-byte
// loads and stores.  Every wait is bounded (Em25Args::wait_ns): one that runs out
// sets the control block's error word and the block leaves the kernel.
//
// What bounds it: 630 x 70 x 330 cells move 0.52 GB a half-step, 78 us at the
// copy bandwidth.  One column a thread with a halo on all sides (32 x 4 columns)
// took 133 + 157 us: it issued 188 instructions a cell -- the waits, the barrier,
// addresses and single-word accesses of every plane -- and staged 1.9 words for a
// word of a neighbouring field.  Four columns a thread share the first and move
// 16 bytes an access (65 instructions a cell); the one-sided halo of 32 x 16
// columns stages 1.2 words: 107 + 135 us, 0.252 against 0.299 ms a step.  What is
// left is the latency of a plane's chain at 12 warps an SM: rings of 3 and 5
// planes (16 and 8 warps) ran 0.009 and 0.020 ms longer, blocks of 8 rows 0.001.  The
// x and z strips' variables, loaded where they were used, cost 0.077 ms.
constexpr int BX = 32;
constexpr int VW = BX + 4;  // floats of a staged row with its halo
constexpr int kRing = 4;  // staged planes per block
constexpr int kThreadsSM = 384;  // resident threads an SM the kernels are compiled for

// Places in a stage (floats), every box on a 128-byte boundary.
template <int TZ>
struct Stage {
  static constexpr int F = (TZ + 1) * VW;               // one field with the halo
  static constexpr int halo = 3 * F;
  static constexpr int own = (halo + 31) & ~31;         // three fields of the own cells
  static constexpr int O = TZ * BX;                     // one of them
  static constexpr int psi = own + 3 * O;               // the two y-strip memory variables of the kernel
  static constexpr int ytab = psi + 2 * O;              // the y table around the plane: 6 rows x 4 entries from j & ~3
  static constexpr int size = ytab + 32;
};

__device__ __forceinline__ float& el(float4& v, int e) { return (&v.x)[e]; }
__device__ __forceinline__ float el(const float4& v, int e) { return (&v.x)[e]; }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// Whether every column of the block at (i0, k0) lies off the x and z CPML
// strips and two cells or more inside the grid (off every Dirichlet face of
// E and H: 1 <= i <= NX - 3, 1 <= k <= NZ - 3).
__device__ __forceinline__ bool block_interior(int i0, int k0, int TZ, int NX, int NZ, int W) {
  return i0 >= max(W, 1) && i0 + BX - 1 <= min(NX - W - 1, NX - 3) && k0 >= max(W, 1) &&
         k0 + TZ - 1 <= min(NZ - W - 1, NZ - 3);
}

__device__ void em25_wait_failed(const Em25Args& a, uint64_t* full, int n, int np) {
  atomicExch(const_cast<int*>(&a.io.ctl->err), 1);
  const int issued = min(np, n + kRing);
  for (int m = n; m < issued; ++m) tma::bar_wait(full + m % kRing, (m / kRing) & 1, a.wait_ns);
}

// Every product, fused product and sum of an update names its rounding, and
// the form a curl's sum takes is a property of the cell alone: where a group of
// 32 x 4 columns lies off the strips and faces (block_interior) one derivative's
// product is fused into the sum, elsewhere both derivatives are rounded first.
// So a cell's bits depend neither on the rows of its block nor on the march that
// advances it.  Near a source the two derivatives cancel, and the rounding error
// either form leaves there stays in H: with the form chosen by whole blocks of 16
// rows, the final Hz of a 630 x 70 x 330 shot was 4.7e-6 from 64 bits instead
// of 3.0e-6.  d ik = w rounded, v the other derivative.
__device__ __forceinline__ float sum2(bool fused, float d, float ik, float w, float v) {
  return fused ? __fmaf_rn(d, ik, v) : __fadd_rn(w, v);
}

// The recursion of four cells' memory variable p <- b p + ad d and what it adds
// to their derivative v; cells outside the loop (act) keep theirs.
template <bool ALL>
__device__ __forceinline__ float4 recur(float4 p, float b, float ad, const float4& d, float4& v, unsigned act) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float m = __fmaf_rn(ad, el(d, e), __fmul_rn(b, el(p, e)));
    if (ALL || (act >> e & 1u)) {
      el(p, e) = m;
      el(v, e) = __fadd_rn(el(v, e), m);
    }
  }
  return p;
}
// The x-strip cells of a thread: the cells of both strips lie back to back at a
// row's memory, from `at` less their element on, those of `high` (the high
// strip's, in a thread with cells of both) `gap` places further down.
struct XCells {
  unsigned in, high;
  int at, gap;
  __device__ __forceinline__ XCells(int i, int NX, int W, bool on) {
    in = high = 0;
    gap = NX - 2 * W;
    at = i < W ? i : i - gap;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (on && i + e < NX && in_strip(i + e, NX, W)) in |= 1u << e;
      if (i < W && i + e >= NX - W) high |= 1u << e;
    }
  }
  __device__ __forceinline__ int place(int e) const { return at + e - (high >> e & 1u ? gap : 0); }
  __device__ __forceinline__ float4 load(const float* row) const {
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (in >> e & 1u) el(p, e) = row[place(e)];
    return p;
  }
  // the recursion as recur's, in the cells of act
  __device__ __forceinline__ void recur(float* row, const float4& p, const float4& b, const float4& ad, const float4& d,
                                        float4& v, unsigned act) const {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (in & act & (1u << e)) {
        const float m = __fmaf_rn(el(ad, e), el(d, e), __fmul_rn(el(b, e), el(p, e)));
        row[place(e)] = m;
        el(v, e) = __fadd_rn(el(v, e), m);
      }
  }
};

template <int TZ>
__global__ void __launch_bounds__(8 * TZ, kThreadsSM / (8 * TZ)) em25_h_tma_kernel(const __grid_constant__ Em25Args a, int rel) {
  using S = Stage<TZ>;
  extern __shared__ __align__(128) unsigned char stage_raw[];
  float* const stage = tma::aligned_stage(stage_raw);
  __shared__ __align__(8) uint64_t full[kRing];
  const Ctl* ctl = a.io.ctl;
  const int t = ctl->base + rel;
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && t > ctl->run_start) {
    const float* ch[3] = {a.Ex, a.Ey, a.Ez};
    gather_receivers<3>(a.io.rec, a.io.nrec, a.io.traces, t - 1, ch, a.P, a.NY, true);
  }
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int i0 = blockIdx.x * BX, k0 = blockIdx.y * TZ;
  const int NX = a.NX, NY = a.NY, NZ = a.NZ, P = a.P, W = a.W;
  const int seg = (NY + a.ysplit - 1) / a.ysplit;
  const int j0 = blockIdx.z * seg, j1 = min(NY - 1, j0 + seg);  // every H loop runs over j <= NY-2
  if (j0 >= j1) return;  // the whole block
  const int np = j1 - j0 + 1;  // the segment's planes and the next one (its E only)
  if (tid == 0) {
    for (int q = 0; q < kRing; ++q) tma::bar_init(full + q, 1);
    tma::fence_bar_init();
  }
  __syncthreads();
  auto issue = [&](int n) {
    float* st = stage + (n % kRing) * S::size;
    uint64_t* bar = full + n % kRing;
    const int j = j0 + n;
    const bool own = j < j1, ys = own && in_strip(j, NY, W);
    tma::bar_arrive_expect(bar, (S::halo + (own ? 3 * S::O + 24 : 0) + (ys ? 2 * S::O : 0)) * 4u + a.stall_tx);
    tma::load_4d(st, &a.tm_halo, bar, i0, j, k0, 0);  // Ex Ey Ez
    if (own) {
      tma::load_4d(st + S::own, &a.tm_own, bar, i0, j, k0, 3);  // Hx Hy Hz
      tma::load_2d(st + S::ytab, &a.tm_ytab, bar, j & ~3, 0);
    }
    if (ys) tma::load_4d(st + S::psi, &a.tm_ypsi_e, bar, i0, strip_idx(j, NY, W), k0, 0);  // dEz_dy dEx_dy
  };
  if (tid == 0)
    for (int n = 0; n < min(kRing, np); ++n) issue(n);

  const int i = i0 + 4 * tx, k = k0 + ty;
  const bool rowc = k <= NZ - 2 && i <= NX - 2;
  const int ic = rowc ? i : 0, kc = rowc ? k : 0;
  const bool interior = block_interior(i0, k0, TZ, NX, NZ, W);
  const bool plain = block_interior(i0, k0 + (ty & ~3), 4, NX, NZ, W);  // this warp's 32 x 4 columns are
  unsigned act = 0, i_lo = 0, i_hi = 0;  // cells the loops update, i = 0, i = NX - 2
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (rowc && i + e <= NX - 2) act |= 1u << e;
    if (i + e == 0) i_lo |= 1u << e;
    if (i + e == NX - 2) i_hi |= 1u << e;
  }
  const bool zsc = rowc && in_strip(k, NZ, W);
  const int zsi = zsc ? strip_idx(k, NZ, W) : 0;
  const XCells xc(i, NX, W, rowc);
  const float4 ikx = ld4(a.X.ik + ic), adx = ld4(a.X.ad + ic), bx = ld4(a.X.b + ic);
  const float ikz = a.Z.ik[kc], adz = a.Z.ad[kc], bz = a.Z.b[kc];
  const float ikzh = a.Z.ikh[kc], adzh = a.Z.adh[kc], bzh = a.Z.bh[kc];
  const float dbH = a.dbH;
  // Dirichlet faces of the previous H that do not depend on j
  const unsigned fxc = (k == 0 || k == NZ - 2) ? 15u : i_lo, fyc = (k == 0 || k == NZ - 2) ? 15u : i_lo | i_hi,
                 fzc = k == 0 ? 15u : i_lo | i_hi;
  const int hc = ty * VW + 4 * tx;  // own cells in a tile with halo
  const int oc = 4 * tid;           // own cells in an own-cells tile
  size_t c = ((size_t)kc * NY + j0) * P + ic;
  // The march, compiled twice: for blocks of interior columns only (I: no x
  // or z memory variables, no faces) and for the others.
  auto march = [&](auto interior_tag) {
    constexpr bool I = decltype(interior_tag)::value;
    const bool row = I || rowc, zs = !I && zsc, xs = !I && xc.in != 0, fused = I || plain;
    float4 ex, ez;  // of plane j, carried from the step before
    // the x and z memory variables of plane j, loaded a step ahead
    const size_t zo = ((size_t)zsi * NY + j0) * P + i, xo = ((size_t)k * NY + j0) * (2 * W);
    float *mz0 = a.mEy_z + zo, *mz1 = a.mEx_z + zo, *mx0 = a.mEz_x + xo, *mx1 = a.mEy_x + xo;
    float4 z0, z1, x0, x1;
    auto load_strips = [&] {
      if (zs) { z0 = ld4(mz0); z1 = ld4(mz1); }
      if (xs) { x0 = xc.load(mx0); x1 = xc.load(mx1); }
    };
    load_strips();
    bool ok = tma::bar_wait(full, 0, a.wait_ns);
    ex = ld4(stage + hc);
    ez = ld4(stage + 2 * S::F + hc);
    for (int n = 0; n < j1 - j0; ++n, c += P) {
      const int j = j0 + n;
      if (ok) ok = tma::bar_wait(full + (n + 1) % kRing, ((n + 1) / kRing) & 1, a.wait_ns);
      if (ok && row) {
        const float* E = stage + (n % kRing) * S::size;  // Ex Ey Ez of plane j, with the halo
        const float* En = stage + ((n + 1) % kRing) * S::size;  // plane j + 1
        const float* H = E + S::own;                            // Hx Hy Hz of the own cells
        const bool ys = in_strip(j, NY, W);
        const float* yt = E + S::ytab + (j & 3);  // rows ik ad b ikh adh bh of the y table
        const float iky = yt[0], ikyh = yt[12];
        const float4 exn = ld4(En + hc), ezn = ld4(En + 2 * S::F + hc);
        const float4 ey = ld4(E + S::F + hc), eyz = ld4(E + S::F + hc + VW), exz = ld4(E + hc + VW);
        const float ezr = E[2 * S::F + hc + 4], eyr = E[S::F + hc + 4];
        float4 dy, d, v, w;
        {  // Hx, :904-917
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(dy, e) = el(ez, e) - el(ezn, e);  // dEz/dy
            el(d, e) = el(eyz, e) - el(ey, e);   // dEy/dz
            el(v, e) = __fmul_rn(el(dy, e), ikyh);
            el(w, e) = __fmul_rn(el(d, e), ikzh);
          }
          if (ys) {
            const size_t my = ((size_t)k * (2 * W) + strip_idx(j, NY, W)) * P + i;
            st4(a.mEz_y + my, recur<I>(ld4(E + S::psi + oc), yt[20], yt[16], dy, v, act));
          }
          if (zs) st4(mz0, recur<I>(z0, bzh, adzh, d, w, act));
          float4 h = ld4(H + oc);
          const unsigned f = j == 0 || j == NY - 2 ? 15u : fxc;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float o = (I ? (j == 0 || j == NY - 2) : (f >> e & 1u)) ? 0.f : el(h, e);
            if (I || (act >> e & 1u)) el(h, e) = __fmaf_rn(dbH, sum2(fused, el(d, e), ikzh, el(w, e), el(v, e)), o);
          }
          st4(a.Hx + c, h);
        }
        {  // Hy, :925-938
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(dy, e) = el(ex, e) - el(exz, e);                                // dEx/dz
            el(d, e) = (e < 3 ? el(ez, e < 3 ? e + 1 : e) : ezr) - el(ez, e);  // dEz/dx
            el(v, e) = __fmul_rn(el(dy, e), ikz);
            el(w, e) = __fmul_rn(el(d, e), el(ikx, e));
          }
          if (zs) st4(mz1, recur<I>(z1, bz, adz, dy, v, act));
          if (xs) xc.recur(mx0, x0, bx, adx, d, w, act);
          float4 h = ld4(H + S::O + oc);
          const unsigned f = j == 0 ? 15u : fyc;  // Hy face j=NY-1 is outside the loop
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float o = (I ? j == 0 : (f >> e & 1u)) ? 0.f : el(h, e);
            if (I || (act >> e & 1u)) el(h, e) = __fmaf_rn(dbH, sum2(fused, el(dy, e), ikz, el(v, e), el(w, e)), o);
          }
          st4(a.Hy + c, h);
        }
        if (I || k >= 1) {  // Hz, :946-960
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(dy, e) = el(exn, e) - el(ex, e);                                // dEx/dy
            el(d, e) = el(ey, e) - (e < 3 ? el(ey, e < 3 ? e + 1 : e) : eyr);  // dEy/dx
            el(v, e) = __fmul_rn(el(dy, e), iky);
            el(w, e) = __fmul_rn(el(d, e), el(ikx, e));
          }
          if (ys) {
            const size_t my = ((size_t)k * (2 * W) + strip_idx(j, NY, W)) * P + i;
            st4(a.mEx_y + my, recur<I>(ld4(E + S::psi + S::O + oc), yt[8], yt[4], dy, v, act));
          }
          if (xs) xc.recur(mx1, x1, bx, adx, d, w, act);
          float4 h = ld4(H + 2 * S::O + oc);
          const unsigned f = j == 0 || j == NY - 2 ? 15u : fzc;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float o = (I ? (j == 0 || j == NY - 2) : (f >> e & 1u)) ? 0.f : el(h, e);
            if (I || (act >> e & 1u)) el(h, e) = __fmaf_rn(dbH, sum2(fused, el(d, e), el(ikx, e), el(w, e), el(v, e)), o);
          }
          st4(a.Hz + c, h);
        }
        ex = exn;
        ez = ezn;
        if (!I && n + 1 < j1 - j0) {
          mz0 += P; mz1 += P; mx0 += 2 * W; mx1 += 2 * W;
          load_strips();
        }
      }
      if (!__syncthreads_and(ok)) {  // every thread is done with plane n (or a wait ran out)
        if (tid == 0) em25_wait_failed(a, full, n, np);
        break;
      }
      if (tid == 0 && n + kRing < np) {
        tma::fence_async_smem();
        issue(n + kRing);
      }
    }
  };
  if (interior) march(std::true_type{});
  else march(std::false_type{});
}

template <int TZ>
__global__ void __launch_bounds__(8 * TZ, kThreadsSM / (8 * TZ)) em25_e_tma_kernel(const __grid_constant__ Em25Args a, int rel) {
  using S = Stage<TZ>;
  extern __shared__ __align__(128) unsigned char stage_raw[];
  float* const stage = tma::aligned_stage(stage_raw);
  __shared__ __align__(8) uint64_t full[kRing];
  const int t = a.io.ctl->base + rel;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int i0 = blockIdx.x * BX, k0 = blockIdx.y * TZ;
  const int NX = a.NX, NY = a.NY, NZ = a.NZ, P = a.P, W = a.W;
  const int seg = (NY + a.ysplit - 1) / a.ysplit;
  const int j0 = blockIdx.z * seg, j1 = min(NY, j0 + seg);
  const int slot = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  float norm = 0.0f;
  if (j0 >= j1) {  // the whole block
    block_norm_to_slot(norm, a.io.slots, slot);
    return;
  }
  const int np = j1 - j0;
  if (tid == 0) {
    for (int q = 0; q < kRing; ++q) tma::bar_init(full + q, 1);
    tma::fence_bar_init();
  }
  __syncthreads();
  auto issue = [&](int n) {
    float* st = stage + (n % kRing) * S::size;
    uint64_t* bar = full + n % kRing;
    const int j = j0 + n;
    const bool ys = in_strip(j, NY, W);
    tma::bar_arrive_expect(bar, (S::halo + 3 * S::O + 24 + (ys ? 2 * S::O : 0)) * 4u + a.stall_tx);
    tma::load_4d(st, &a.tm_halo, bar, i0 - 4, j, k0 - 1, 3);  // Hx Hy Hz
    tma::load_4d(st + S::own, &a.tm_own, bar, i0, j, k0, 0);  // Ex Ey Ez
    tma::load_2d(st + S::ytab, &a.tm_ytab, bar, j & ~3, 0);
    if (ys) tma::load_4d(st + S::psi, &a.tm_ypsi_h, bar, i0, strip_idx(j, NY, W), k0, 0);  // dHz_dy dHx_dy
  };
  if (tid == 0)
    for (int n = 0; n < min(kRing, np); ++n) issue(n);

  const int i = i0 + 4 * tx, k = k0 + ty;
  const bool rowc = i < NX && k < NZ;
  const int ic = rowc ? i : 0, kc = rowc ? k : 0;
  const bool interior = block_interior(i0, k0, TZ, NX, NZ, W);
  const bool plain = block_interior(i0, k0 + (ty & ~3), 4, NX, NZ, W);  // this warp's 32 x 4 columns are
  const bool krow = k >= 1 && k <= NZ - 2;
  // cells each loop updates, the Dirichlet faces off j
  unsigned uX = 0, uY = 0, uZ = 0, fX = 0, fY = 0, fZ = 0;
  const size_t pc = (size_t)kc * P + ic;
  float4 caX = make_float4(0.f, 0.f, 0.f, 0.f), cbX = caX, caY = caX, cbY = caX, caZ = caX, cbZ = caX;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int ie = i + e;
    if (!rowc || ie >= NX) continue;
    if (krow && ie <= NX - 2) {
      uX |= 1u << e;
      el(caX, e) = a.caEx[pc + e];
      el(cbX, e) = a.cbEx[pc + e];
    }
    if (krow && ie >= 1 && ie <= NX - 2) {  // (4 c(i,k) + c(i-1,k) + c(i,k-1)) / 6, :1004-1006
      uY |= 1u << e;
      el(caY, e) = (4.f * a.caEy[pc + e] + a.caEy[pc + e - 1] + a.caEy[pc + e - P]) / 6.f;
      el(cbY, e) = (4.f * a.cbEy[pc + e] + a.cbEy[pc + e - 1] + a.cbEy[pc + e - P]) / 6.f;
    }
    if (k <= NZ - 2 && ie >= 1 && ie <= NX - 2) {  // (4 c(i,k) + c(i-1,k) + c(i,k+1)) / 6, :1026-1028
      uZ |= 1u << e;
      el(caZ, e) = (4.f * a.caEz[pc + e] + a.caEz[pc + e - 1] + a.caEz[pc + e + P]) / 6.f;
      el(cbZ, e) = (4.f * a.cbEz[pc + e] + a.cbEz[pc + e - 1] + a.cbEz[pc + e + P]) / 6.f;
    }
    if (ie == 0 || ie == NX - 2 || k == 0 || k == NZ - 1) fX |= 1u << e;
    if (ie == 0 || ie == NX - 1 || k == 0 || k == NZ - 1) fY |= 1u << e;
    if (ie == 0 || ie == NX - 1 || k == 0 || k == NZ - 2) fZ |= 1u << e;
  }
  const bool zsc = rowc && in_strip(k, NZ, W);
  const int zsi = zsc ? strip_idx(k, NZ, W) : 0;
  const XCells xc(i, NX, W, rowc);
  const float4 ikxh = ld4(a.X.ikh + ic), adxh = ld4(a.X.adh + ic), bxh = ld4(a.X.bh + ic);
  const float ikz = a.Z.ik[kc], adz = a.Z.ad[kc], bz = a.Z.b[kc];
  const float ikzh = a.Z.ikh[kc], adzh = a.Z.adh[kc], bzh = a.Z.bh[kc];
  const int hc = (ty + 1) * VW + 4 * tx + 4;
  const int oc = 4 * tid;
  size_t c = ((size_t)kc * NY + j0) * P + ic;
  float4 phx = make_float4(0.f, 0.f, 0.f, 0.f), phz = phx;  // Hx, Hz of the plane before
  if (rowc && j0 >= 1) {
    phx = __ldg(reinterpret_cast<const float4*>(a.Hx + c - P));
    phz = __ldg(reinterpret_cast<const float4*>(a.Hz + c - P));
  }
  const bool src_col = rowc && k == a.io.sk && a.io.si >= i && a.io.si < i + 4;
  // compiled twice, as the H kernel's march
  auto march = [&](auto interior_tag) {
    constexpr bool I = decltype(interior_tag)::value;
    const bool row = I || rowc, zs = !I && zsc, xs = !I && xc.in != 0, fused = I || plain;
    // the x and z memory variables of plane j, loaded a step ahead
    const size_t zo = ((size_t)zsi * NY + j0) * P + i, xo = ((size_t)k * NY + j0) * (2 * W);
    float *mz0 = a.mHy_z + zo, *mz1 = a.mHx_z + zo, *mx0 = a.mHz_x + xo, *mx1 = a.mHy_x + xo;
    float4 z0, z1, x0, x1;
    auto load_strips = [&] {
      if (zs) { z0 = ld4(mz0); z1 = ld4(mz1); }
      if (xs) { x0 = xc.load(mx0); x1 = xc.load(mx1); }
    };
    load_strips();
    for (int n = 0; n < np; ++n, c += P) {
      const int j = j0 + n;
      const bool ok = tma::bar_wait(full + n % kRing, (n / kRing) & 1, a.wait_ns);
      if (ok && row) {
        const float* H = stage + (n % kRing) * S::size;  // Hx Hy Hz of plane j, with the halo
        const float* E = H + S::own;                     // Ex Ey Ez of the own cells
        const bool ys = in_strip(j, NY, W), mid = j >= 1 && j <= NY - 2;
        const float* yt = H + S::ytab + (j & 3);  // rows ik ad b ikh adh bh of the y table
        const float ikyh = yt[12];
        const float4 hx = ld4(H + hc), hy = ld4(H + S::F + hc), hz = ld4(H + 2 * S::F + hc);
        float4 ex = ld4(E + oc), ey = ld4(E + S::O + oc), ez = ld4(E + 2 * S::O + oc);
        float4 d, f, v, w;
        if ((I || uX) && mid) {  // Ex, :971-984
          const float4 hym = ld4(H + S::F + hc - VW);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(d, e) = el(hz, e) - el(phz, e);  // dHz/dy
            el(f, e) = el(hym, e) - el(hy, e);  // dHy/dz
            el(v, e) = __fmul_rn(el(d, e), ikyh);
            el(w, e) = __fmul_rn(el(f, e), ikz);
          }
          if (ys) {
            const size_t my = ((size_t)k * (2 * W) + strip_idx(j, NY, W)) * P + i;
            st4(a.mHz_y + my, recur<I>(ld4(H + S::psi + oc), yt[20], yt[16], d, v, uX));
          }
          if (zs) st4(mz0, recur<I>(z0, bz, adz, f, w, uX));
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (I || (uX >> e & 1u)) el(ex, e) = __fmaf_rn(el(caX, e), el(ex, e), __fmul_rn(el(cbX, e), sum2(fused, el(f, e), ikz, el(w, e), el(v, e))));
        }
        const float4 hxm = ld4(H + hc - VW);
        if ((I || uY) && j <= NY - 2) {  // Ey, :988-1007
          const float hzl = H[2 * S::F + hc - 1];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(d, e) = (e > 0 ? el(hz, e > 0 ? e - 1 : 0) : hzl) - el(hz, e);  // dHz/dx
            el(f, e) = el(hx, e) - el(hxm, e);                                 // dHx/dz
            el(v, e) = __fmul_rn(el(d, e), el(ikxh, e));
            el(w, e) = __fmul_rn(el(f, e), ikzh);
          }
          if (xs) xc.recur(mx0, x0, bxh, adxh, d, v, uY);
          if (zs) st4(mz1, recur<I>(z1, bzh, adzh, f, w, uY));
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (I || (uY >> e & 1u)) el(ey, e) = __fmaf_rn(el(caY, e), el(ey, e), __fmul_rn(el(cbY, e), sum2(fused, el(d, e), el(ikxh, e), el(v, e), el(w, e))));
        }
        if ((I || uZ) && mid) {  // Ez, :1015-1029
          const float hyl = H[S::F + hc - 1];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(d, e) = el(phx, e) - el(hx, e);                                 // dHx/dy
            el(f, e) = el(hy, e) - (e > 0 ? el(hy, e > 0 ? e - 1 : 0) : hyl);  // dHy/dx
            el(v, e) = __fmul_rn(el(d, e), ikyh);
            el(w, e) = __fmul_rn(el(f, e), el(ikxh, e));
          }
          if (ys) {
            const size_t my = ((size_t)k * (2 * W) + strip_idx(j, NY, W)) * P + i;
            st4(a.mHx_y + my, recur<I>(ld4(H + S::psi + S::O + oc), yt[20], yt[16], d, v, uZ));
          }
          if (xs) xc.recur(mx1, x1, bxh, adxh, f, w, uZ);
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (I || (uZ >> e & 1u)) el(ez, e) = __fmaf_rn(el(caZ, e), el(ez, e), __fmul_rn(el(cbZ, e), sum2(fused, el(f, e), el(ikxh, e), el(w, e), el(v, e))));
        }
        if (src_col && j == a.io.sj) {  // :1033-1035
          const float sx = a.io.src[t], sy = a.io.src[a.io.nstep + t], sz = a.io.src[2 * a.io.nstep + t];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (i + e == a.io.si) {
              el(ex, e) += sx;
              el(ey, e) += sy;
              el(ez, e) += sz;
            }
        }
        const bool jx = j == 0 || j == NY - 1, jy = j == 0 || j == NY - 2;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (jx || (!I && (fX >> e & 1u))) el(ex, e) = 0.f;  // :1038-1043
          if (jy || (!I && (fY >> e & 1u))) el(ey, e) = 0.f;  // :1045-1050
          if (jx || (!I && (fZ >> e & 1u))) el(ez, e) = 0.f;  // :1052-1057
          norm = fmaxf(norm, norm_monitor(el(ex, e), el(ey, e), el(ez, e)));
        }
        st4(a.Ex + c, ex);
        st4(a.Ey + c, ey);
        st4(a.Ez + c, ez);
        phx = hx;
        phz = hz;
        if (!I && n + 1 < np) {
          mz0 += P; mz1 += P; mx0 += 2 * W; mx1 += 2 * W;
          load_strips();
        }
      }
      if (!__syncthreads_and(ok)) {
        if (tid == 0) em25_wait_failed(a, full, n, np);
        break;
      }
      if (tid == 0 && n + kRing < np) {
        tma::fence_async_smem();
        issue(n + kRing);
      }
    }
  };
  if (interior) march(std::true_type{});
  else march(std::false_type{});
  block_norm_to_slot(norm, a.io.slots, slot);
}

// Zero the H Dirichlet faces (:1059-1078) in memory.
__global__ void em25_hfaces_kernel(Em25Args a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y * blockDim.y + threadIdx.y;
  const int NX = a.NX, NY = a.NY, NZ = a.NZ, P = a.P;
  if (i >= NX || k >= NZ) return;
  const bool fx = (i == 0) || (i == NX - 1) || (k == 0) || (k == NZ - 2);
  const bool fy = (i == 0) || (i == NX - 2) || (k == 0) || (k == NZ - 2);
  const bool fz = (i == 0) || (i == NX - 2) || (k == 0) || (k == NZ - 1);
  for (int j = 0; j < NY; ++j) {
    const size_t c = ((size_t)k * NY + j) * P + i;
    if (fx || j == 0 || j == NY - 2) a.Hx[c] = 0.f;
    if (fy || j == 0 || j == NY - 1) a.Hy[c] = 0.f;
    if (fz || j == 0 || j == NY - 2) a.Hz[c] = 0.f;
  }
}

__global__ void em25_finalize_kernel(Em25Args a, int t_last) {
  const float* ch[3] = {a.Ex, a.Ey, a.Ez};
  gather_receivers<3>(a.io.rec, a.io.nrec, a.io.traces, t_last, ch, a.P, a.NY, true);
}

}  // namespace

// Rows of a block: the most of 16, 8, 4 with two blocks an SM (100 x 60 x 81
// cells: 21.5 us a step in blocks of 16 rows, 28 in those of 32 x 4 single
// columns; 44 x 36 x 40, too small for either: 16 against 18).
static int em25_rows(int NX, int NZ, int ysplit) {
  for (int tz = 16; tz > 4; tz /= 2)
    if ((long)((NX + BX - 1) / BX) * ((NZ + tz - 1) / tz) * ysplit >= 2 * 152) return tz;
  return 4;
}

Launch em25_launch(const Em25Args& a) {
  const int tz = em25_rows(a.NX, a.NZ, a.ysplit);
  Launch L;
  L.block = dim3(8 * tz, 1, 1);
  L.grid = dim3((a.NX + BX - 1) / BX, (a.NZ + tz - 1) / tz, a.ysplit);
  L.nslots = L.grid.x * L.grid.y * L.grid.z;
  return L;
}

template <int TZ>
static constexpr size_t kStageBytes = kRing * Stage<TZ>::size * sizeof(float) + tma::kStageSlack;

void em25_half1(const Em25Args& a, const Launch& L, int rel, cudaStream_t s) {
  switch (L.block.x / 8) {
    case 16: em25_h_tma_kernel<16><<<L.grid, L.block, kStageBytes<16>, s>>>(a, rel); break;
    case 8: em25_h_tma_kernel<8><<<L.grid, L.block, kStageBytes<8>, s>>>(a, rel); break;
    default: em25_h_tma_kernel<4><<<L.grid, L.block, kStageBytes<4>, s>>>(a, rel);
  }
}

void em25_half2(const Em25Args& a, const Launch& L, int rel, cudaStream_t s) {
  switch (L.block.x / 8) {
    case 16: em25_e_tma_kernel<16><<<L.grid, L.block, kStageBytes<16>, s>>>(a, rel); break;
    case 8: em25_e_tma_kernel<8><<<L.grid, L.block, kStageBytes<8>, s>>>(a, rel); break;
    default: em25_e_tma_kernel<4><<<L.grid, L.block, kStageBytes<4>, s>>>(a, rel);
  }
}

bool em25_make_maps(Em25Args& a, size_t field_stride, const float* ytab) {
  const int tz = em25_rows(a.NX, a.NZ, a.ysplit);
  // stages of 16 rows exceed the default 48 KB
  if (cudaFuncSetAttribute(em25_h_tma_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageBytes<16>) !=
          cudaSuccess ||
      cudaFuncSetAttribute(em25_e_tma_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageBytes<16>) !=
          cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (!(encode_field_map(&a.tm_halo, a.Ex, a.NX, a.NY, a.NZ, a.P, field_stride, 6, VW, tz + 1, 3) &&
        encode_field_map(&a.tm_own, a.Ex, a.NX, a.NY, a.NZ, a.P, field_stride, 6, BX, tz, 3)))
    return false;
  // the y-strip memory variables (layout [k][2W][P]) each kernel reads: two arrays
  auto ypsi = [&](CUtensorMap* m, float* m0, float* m1) {
    const size_t d = (size_t)((char*)m1 - (char*)m0);
    if (d % 16) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)a.NX, (cuuint64_t)(2 * a.W), (cuuint64_t)a.NZ, 2};
    const cuuint64_t strides[3] = {(cuuint64_t)a.P * 4, (cuuint64_t)2 * a.W * a.P * 4, (cuuint64_t)d};
    const cuuint32_t box[4] = {BX, 1, (cuuint32_t)tz, 2};
    return encode_tiled(m, m0, 4, dims, strides, box);
  };
  if (!ypsi(&a.tm_ypsi_e, a.mEz_y, a.mEx_y) || !ypsi(&a.tm_ypsi_h, a.mHz_y, a.mHx_y)) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)axis_stride(a.NY), 6};
  const cuuint64_t strides[1] = {(cuuint64_t)axis_stride(a.NY) * 4};
  const cuuint32_t box[2] = {4, 6};
  return encode_tiled(&a.tm_ytab, (void*)ytab, 2, dims, strides, box);
}

void em25_finalize(const Em25Args& a, int t_last, cudaStream_t s) {
  dim3 b(32, 8), g((a.NX + 31) / 32, (a.NZ + 7) / 8);
  em25_hfaces_kernel<<<g, b, 0, s>>>(a);
  em25_finalize_kernel<<<1, 256, 0, s>>>(a, t_last);
}

}  // namespace sfd

// Streaming electromag2c runs: kC2Halo steps of the complex scheme (em2c.cu) a
// launch, every launch reading one copy of the state and writing the other.
//
// The tiles are electromag2's (em2_tile.cuh, em2_stream.cu) at two cells a lane:
// a CTA loads its frame -- the owned cells and kC2Halo cells of halo --, holds
// the six field planes in registers (a warp RB whole rows of 64 columns) and the
// eight coefficient planes in shared memory, advances them by up to kC2Halo
// steps and writes the owned cells.  Neighbours along x are a shuffle away,
// along z in the same thread but for the first and last row of a warp, which
// pass through shared memory.  Loop bounds and Dirichlet planes are coefficient
// values.  A tile whose strips leave no room for the coefficients (npml above
// some 40 cells) reads them from L2 every step instead.
//
// What bounds it: the state of 1040 x 540 cells and its coefficients (31 MB) stay
// in L2, and the two-kernel step waited on it twice a step: 13.5 us a step, 256
// steps 3.45 ms.  Here a step takes 8.3 us, 256 steps 2.12 ms.  A launch of
// four steps lasts as long as its slowest tile, one of the grid's edge: 10 us
// to load the frame (287 KB, L2 rate), 3.3 us a step (1.8 us off the strips),
// 4 us to store.  Five rows a warp make 152 tiles of that grid, one wave; four
// rows (190 tiles) take 2.12 ms as well, three 2.5 ms.  Frames of 26 warps of
// three rows and 20 of four spill and take 4.7 and 3.3 ms.
#include <algorithm>

#include "em2_tile.cuh"

namespace sfd {

using namespace res;
using tile2::copies_wait;
using tile2::copy8;
using tile2::max_nan;

namespace {

constexpr int kCC = 64, kWarps = 16, kThreads = 32 * kWarps;  // frame columns, warps
constexpr int kMaxRows = 5;                                   // most rows a warp
// places in c2_smem (floats): x tables ik ad b ikh adh bh, each warp's first Ex
// row and last Hy row (re, im), row tables [rows][8] ik b ad - ikh bh adh -, then
// the z strips' rows [][4][64] (dEx_dz, dHy_dz, re and im), the x strips' lanes
// [rows][4][2 nxl] (dEz_dx, dHy_dx) and the coefficients [rows][8][64]
constexpr int kOE = 6 * kCC, kOHc = kOE + 2 * kWarps * kCC, kORTc = kOHc + 2 * kWarps * kCC;
// The cost of a tile's barriers and launch, in rows a warp (0.5 to 5 measured alike).
constexpr double kC2TileCost = 2.0;
constexpr int kMaxRec = 256;  // receivers a tile lists; with more it scans them all every step

extern __shared__ __align__(16) float c2_smem[];

struct cf2 {  // two complex cells
  float2 r, i;
};
__device__ __forceinline__ float& el(float2& v, int e) { return (&v.x)[e]; }
__device__ __forceinline__ float el(const float2& v, int e) { return (&v.x)[e]; }
__device__ __forceinline__ float2& part(cf2& v, int q) { return q ? v.i : v.r; }
__device__ __forceinline__ float2 lds(int o) { return *reinterpret_cast<const float2*>(c2_smem + o); }
__device__ __forceinline__ void sts(int o, float2 v) { *reinterpret_cast<float2*>(c2_smem + o) = v; }
// Tiles of uniform size: ntx columns of at most 56 cells (one of up to 64), nbz
// bands of at most kWarps RB - 2 kC2Halo rows (one of up to kWarps RB).
__host__ __device__ inline int cut_x(int NX, int c, int ntx) {
  const int x = (int)(2 * ((long)((NX + 1) / 2) * c / ntx));
  return x < NX ? x : NX;
}
__host__ __device__ inline int cut_z(int NZ, int r, int nbz) { return (int)((long)NZ * r / nbz); }

// A tile's frame: its bounds, the strip cells in it and the places of its arrays.
struct C2Frame {
  int x0, x1, z0, z1;       // owned cells
  int bx, bz, xend, kend;   // frame
  int R;                    // frame rows in whole warps
  int zlo, zh0, zn;         // rows of the low z strip, first row of the high one, rows of both
  int xlo, xh0, nxl;        // lanes below xlo and from xh0 on hold an x-strip cell; their number
  int oD, oS, oX, oC, end;  // lanes off the x strips, z and x memory variables, coefficients, their end (floats)
};
__host__ __device__ inline int imin(int a, int b) { return a < b ? a : b; }
__host__ __device__ inline int imax(int a, int b) { return a > b ? a : b; }
__host__ __device__ inline C2Frame c2_frame(int NX, int NZ, int W, int rb, int ntx, int nbz, int c, int r) {
  C2Frame f;
  f.x0 = cut_x(NX, c, ntx); f.x1 = cut_x(NX, c + 1, ntx); f.z0 = cut_z(NZ, r, nbz); f.z1 = cut_z(NZ, r + 1, nbz);
  f.bx = imax(f.x0 - kC2Halo, 0); f.xend = imin(NX, f.x1 + kC2Halo);
  f.bz = imax(f.z0 - kC2Halo, 0); f.kend = imin(NZ, f.z1 + kC2Halo);
  f.R = (f.kend - f.bz + rb - 1) / rb * rb;
  f.zlo = imax(imin(W, f.kend) - f.bz, 0);
  f.zh0 = imax(NZ - W, f.bz);
  f.zn = f.zlo + imax(f.kend - f.zh0, 0);
  f.xlo = imax((imin(W, f.xend) - f.bx + 1) / 2, 0);
  f.xh0 = imax((NX - W - f.bx) / 2, f.xlo);
  f.nxl = f.xlo + imax((f.xend - f.bx + 1) / 2 - f.xh0, 0);
  f.oD = kORTc + 8 * kWarps * rb;
  f.oS = f.oD + 2 * 32;
  f.oX = f.oS + 4 * kCC * f.zn;
  f.oC = f.oX + 8 * f.R * f.nxl;
  f.end = f.oC + 8 * kCC * f.R;
  return f;
}

struct C2Tile {
  int nrec;
  int first[kThreads];                // of each thread's receivers among ...
  int rec[kMaxRec], next[kMaxRec];    // ... the tile's: receiver << 4 | 2 * row + element, the thread's next one
};

// The fourth power of the stability monitor |sqrt(Ex^2 + Ez^2)| (complex squares,
// :601) where it may be near 1e25, of components scaled by 2^-100, which neither
// over- nor underflows there.
__device__ __forceinline__ float c2_norm4(float xr, float xi, float zr, float zi) {
  const float s = 7.888609e-31f;  // 2^-100
  xr *= s; xi *= s; zr *= s; zi *= s;
  const float wr = xr * xr - xi * xi + zr * zr - zi * zi, wi = 2.0f * (xr * xi + zr * zi);
  return wr * wr + wi * wi;
}

// One tile.  EDGE: the frame holds CPML strip or boundary cells (a cell outside a
// loop's bounds keeps its value, a Dirichlet cell is zeroed after each step).
// XS: it holds x-strip cells.  CS: its coefficients lie in shared memory.
template <int RB, bool EDGE, bool XS, bool CS>
__device__ __forceinline__ void em2c_tile(const Em2cStream& a, C2Tile& G, const C2Frame& f) {
  const Em2cArgs& s0 = a.from;
  const int NX = s0.NX, NZ = s0.NZ, P = s0.P, W = s0.W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bx = f.bx, xend = f.xend, bz = f.bz, kend = f.kend;
  const int i0 = bx + 2 * lane, kb = bz + warp * RB;
  const int nr = min(max(kend - kb, 0), RB);  // frame rows of this warp
  const bool lact = i0 < xend, lown = i0 >= f.x0 && i0 < f.x1;
  const float2 zero2 = make_float2(0.f, 0.f);
  auto oZ = [&](int k) { return f.oS + 4 * kCC * (k < W ? k - bz : f.zlo + k - f.zh0) + 2 * lane; };  // + q kCC
  const bool xsl = XS && nr > 0 && lact && (lane < f.xlo || lane >= f.xh0);
  // + (4 j + q) sX; the other lanes of an x-strip tile read and write a place of their own (zero tables)
  const int sX = xsl ? 2 * f.nxl : 0;
  const int oX = xsl ? f.oX + 4 * sX * RB * warp + 2 * (lane < f.xlo ? lane : lane - f.xh0 + f.xlo) : f.oD + 2 * lane;
  const int oC = f.oC + 8 * kCC * RB * warp + 2 * lane;                        // + (8 j + q) kCC
  const float* const coef[8] = {s0.CAx[0], s0.CAx[1], s0.CBx[0], s0.CBx[1], s0.CAz[0], s0.CAz[1], s0.CBz[0], s0.CBz[1]};

  // Dirichlet planes of Ex and Ez (:585-594)
  auto x_plane = [&](int i, int k) { return i <= NX - 2 && (i == 0 || i == NX - 2 || k == 0 || k == NZ - 1); };
  auto z_plane = [&](int i, int k) { return k <= NZ - 2 && (i == 0 || i == NX - 1 || k == 0 || k == NZ - 2); };

  // ---- load the frame
  cf2 ex[RB], ez[RB], hy[RB];
  unsigned own = 0, hyz = 0;  // owned rows of this lane; cells (bit 2 * row + element) where Hy is a Dirichlet plane
  int src = -1;               // 2 * row + element of the source cell ...
  bool src_x = false, src_z = false;  // ... unless it is a plane's, and its Ex, Ez are stored
#pragma unroll
  for (int j = 0; j < RB; ++j) {
    const int k = kb + j;
    const bool on = j < nr && lact;
    const size_t g = on ? (size_t)k * P + i0 : 0;
    if (CS && warp * RB + j < f.R)
#pragma unroll
      for (int q = 0; q < 8; ++q) copy8(c2_smem + oC + (8 * j + q) * kCC, coef[q] + g, on);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      part(ex[j], q) = on ? *reinterpret_cast<const float2*>(s0.Ex[q] + g) : zero2;
      part(ez[j], q) = on ? *reinterpret_cast<const float2*>(s0.Ez[q] + g) : zero2;
      part(hy[j], q) = on ? *reinterpret_cast<const float2*>(s0.Hy[q] + g) : zero2;
    }
    if (on && k == s0.io.sk && s0.io.si >= i0 && s0.io.si < i0 + 2) {
      src = 2 * j + s0.io.si - i0;
      src_x = s0.io.si <= NX - 2 && !x_plane(s0.io.si, k);
      src_z = k <= NZ - 2 && !z_plane(s0.io.si, k);
    }
    if (on && lown && k >= f.z0 && k < f.z1) own |= 1u << j;
    if (EDGE && on)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (i0 + e == 0 || i0 + e == NX - 2 || k == 0 || k == NZ - 2) hyz |= 1u << (2 * j + e);
  }
  auto zero_hy = [&] {  // :595-598
#pragma unroll
    for (int q = 0; q < 2 * RB; ++q)
      if (hyz >> q & 1u) el(hy[q / 2].r, q & 1) = el(hy[q / 2].i, q & 1) = 0.0f;
  };
  if (EDGE && hyz) zero_hy();
  if (tid == 0) G.nrec = 0;
  G.first[tid] = -1;
  for (int q = tid; q < 4 * kWarps * kCC; q += kThreads) c2_smem[kOE + q] = 0.0f;  // rows past the frame are read as zero
  {
    const float* const xt[6] = {s0.X.ik, s0.X.ad, s0.X.b, s0.X.ikh, s0.X.adh, s0.X.bh};
    for (int q = warp; q < 6; q += kWarps) {
      float2 t = zero2;
#pragma unroll
      for (int e = 0; e < 2; ++e)  // the recursion runs in strip cells only
        if (i0 + e < xend && (q % 3 == 0 || in_strip(i0 + e, NX, W))) {
          el(t, e) = __ldg(xt[q] + i0 + e);
          if (EDGE && q % 3 && (i0 + e > NX - 2 || (q > 3 && i0 + e < 1))) el(t, e) = q % 3 == 2 ? 1.0f : 0.0f;  // ... what no loop advances
        }
      sts(q * kCC + 2 * lane, t);
    }
    const float* const zt[8] = {s0.Z.ik, s0.Z.b, s0.Z.ad, nullptr, s0.Z.ikh, s0.Z.bh, s0.Z.adh, nullptr};
    for (int q = tid; q < 8 * f.R; q += kThreads) {
      const int k = bz + (q >> 3);
      float t = (q & 3) != 3 && k < kend ? __ldg(zt[q & 7] + k) : 0.0f;
      if (EDGE && (q & 3) && (k > NZ - 2 || (q & 4 && k < 1))) t = (q & 3) == 1 ? 1.0f : 0.0f;  // (b, ad) = (1, 0) keeps ...
      c2_smem[kORTc + q] = t;
    }
    if (XS && warp == kWarps - 1) sts(f.oD + 2 * lane, zero2);
  }
  if (EDGE) {
    const float* const zm[4] = {s0.mExz[0], s0.mExz[1], s0.mHyz[0], s0.mHyz[1]};
    const float* const xm[4] = {s0.mEzx[0], s0.mEzx[1], s0.mHyx[0], s0.mHyx[1]};
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      if (j < nr && in_strip(k, NZ, W)) {
        const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i0;
#pragma unroll
        for (int q = 0; q < 4; ++q) sts(oZ(k) + q * kCC, lact ? *reinterpret_cast<const float2*>(zm[q] + zg) : zero2);
      }
      if (xsl)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const bool on = j < nr && i0 + e < NX && in_strip(i0 + e, NX, W);
          const size_t xg = on ? (size_t)k * (2 * W) + strip_idx(i0 + e, NX, W) : 0;
#pragma unroll
          for (int q = 0; q < 4; ++q) c2_smem[oX + (4 * j + q) * sX + e] = on ? xm[q][xg] : 0.0f;
        }
    }
  }
  __syncthreads();
  // ---- receivers of the owned cells, chained to the threads that hold them
  for (int q = tid; q < s0.io.nrec; q += kThreads) {
    const int i = s0.io.rec[3 * q], k = s0.io.rec[3 * q + 2];
    if (i >= f.x0 && i < f.x1 && k >= f.z0 && k < f.z1) {
      const int pos = atomicAdd(&G.nrec, 1);
      if (pos < kMaxRec) {
        G.rec[pos] = q << 4 | (2 * ((k - bz) % RB) + ((i - bx) & 1));
        G.next[pos] = atomicExch(&G.first[32 * ((k - bz) / RB) + (i - bx) / 2], pos);
      }
    }
  }
  auto show_e = [&] {
    sts(kOE + 2 * warp * kCC + 2 * lane, ex[0].r);
    sts(kOE + (2 * warp + 1) * kCC + 2 * lane, ex[0].i);
  };
  if (nr > 0) show_e();
  __syncthreads();
  const bool listed = G.nrec <= kMaxRec;
  const int rec0 = listed ? G.first[tid] : own ? 0 : -1;  // this thread's first receiver; not listed: all are looked at
  if (CS) copies_wait();  // each thread reads only what it copied
  if (CS && EDGE) {  // loop bounds and planes into the coefficients: (1, 0) carries a cell over, (0, 0) holds it at zero
#pragma unroll 1
    for (int j = 0; j < nr; ++j) {
      const int k = kb + j;
      if (!lact || (k >= 1 && k <= NZ - 3 && i0 >= 1 && i0 + 1 <= NX - 3)) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = i0 + e;
        float* c = c2_smem + oC + 8 * j * kCC + e;
        const bool xp = x_plane(i, k), zp = z_plane(i, k);
        if (xp || i > NX - 2 || k < 1 || k > NZ - 2) {
          c[0] = xp ? 0.0f : 1.0f;
          c[kCC] = c[2 * kCC] = c[3 * kCC] = 0.0f;
        }
        if (zp || i > NX - 2 || i < 1 || k > NZ - 2) {
          c[4 * kCC] = zp ? 0.0f : 1.0f;
          c[5 * kCC] = c[6 * kCC] = c[7 * kCC] = 0.0f;
        }
      }
    }
  }

  // dt / mu0; zero at column NX - 1, whose Hy no loop advances
  float2 dbh = make_float2(s0.dbH, s0.dbH);
  if (XS)
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (i0 + e > NX - 2) el(dbh, e) = 0.0f;
  // b m + ad d
  auto next = [](float b, float m, float ad, float d) { return __fmaf_rn(b, m, __fmul_rn(ad, d)); };
  float nrm = 0.0f;
  for (int s = 0; s < a.nsteps; ++s) {
    if (nr > 0) {  // H half-step (:530-549)
      cf2 exb;
      exb.r = lds(kOE + 2 * min(warp + 1, kWarps - 1) * kCC + 2 * lane);
      exb.i = lds(kOE + (2 * min(warp + 1, kWarps - 1) + 1) * kCC + 2 * lane);
      const float2 ik = lds(2 * lane), xa = XS ? lds(kCC + 2 * lane) : zero2, xb = XS ? lds(2 * kCC + 2 * lane) : zero2;
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const float4 rt = lds4(c2_smem + kORTc + 8 * (warp * RB + j));
        const bool zs = EDGE && j < nr && in_strip(kb + j, NZ, W);
        const int oz = zs ? oZ(kb + j) : 0;
        float2 d[2], v[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 en = j < RB - 1 ? part(ex[j < RB - 1 ? j + 1 : j], q) : part(exb, q);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            el(d[q], e) = __fsub_rn(el(en, e), el(part(ex[j], q), e));
            el(v[q], e) = __fmul_rn(el(d[q], e), rt.x);
          }
        }
        if (zs) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float2 p = lds(oz + q * kCC);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              el(p, e) = next(rt.y, el(p, e), rt.z, el(d[q], e));
              el(v[q], e) = __fadd_rn(el(v[q], e), el(p, e));
            }
            sts(oz + q * kCC, p);
          }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 z = part(ez[j], q);
          float2 dd;
          dd.x = __fsub_rn(z.y, z.x);
          dd.y = __fsub_rn(__shfl_down_sync(0xffffffffu, z.x, 1), z.y);
#pragma unroll
          for (int e = 0; e < 2; ++e) el(v[q], e) = __fmaf_rn(el(dd, e), el(ik, e), el(v[q], e));
          if (XS) {
            float2 p = lds(oX + (4 * j + q) * sX);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              el(p, e) = next(el(xb, e), el(p, e), el(xa, e), el(dd, e));
              el(v[q], e) = __fadd_rn(el(v[q], e), el(p, e));
            }
            sts(oX + (4 * j + q) * sX, p);
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) el(part(hy[j], q), e) = __fmaf_rn(el(dbh, e), el(v[q], e), el(part(hy[j], q), e));
        }
      }
      sts(kOHc + 2 * warp * kCC + 2 * lane, hy[RB - 1].r);
      sts(kOHc + (2 * warp + 1) * kCC + 2 * lane, hy[RB - 1].i);
    }
    __syncthreads();
    if (nr > 0) {  // E half-step (:556-576)
      cf2 ht;
      ht.r = lds(kOHc + 2 * max(warp - 1, 0) * kCC + 2 * lane);
      ht.i = lds(kOHc + (2 * max(warp - 1, 0) + 1) * kCC + 2 * lane);
      const float2 ik = lds(3 * kCC + 2 * lane), xa = XS ? lds(4 * kCC + 2 * lane) : zero2,
                   xb = XS ? lds(5 * kCC + 2 * lane) : zero2;
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const int k = kb + j;
        const float4 rt = lds4(c2_smem + kORTc + 8 * (warp * RB + j) + 4);
        const bool zs = EDGE && j < nr && in_strip(k, NZ, W);
        const int oz = zs ? oZ(k) : 0;
        float2 c[8];
        {
          const size_t g = !CS && j < nr && lact ? (size_t)k * P + i0 : 0;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            c[q] = !CS ? __ldg(reinterpret_cast<const float2*>(coef[q] + g)) : lds(oC + (8 * j + q) * kCC);
        }
        cf2 dz, dx;  // the two scaled differences
        float2 d[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 hm = j > 0 ? part(hy[j > 0 ? j - 1 : 0], q) : part(ht, q);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            el(d[q], e) = __fsub_rn(el(part(hy[j], q), e), el(hm, e));
            el(part(dz, q), e) = __fmul_rn(el(d[q], e), rt.x);
          }
        }
        if (zs) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float2 p = lds(oz + (2 + q) * kCC);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              el(p, e) = next(rt.y, el(p, e), rt.z, el(d[q], e));
              el(part(dz, q), e) = __fadd_rn(el(part(dz, q), e), el(p, e));
            }
            sts(oz + (2 + q) * kCC, p);
          }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 h = part(hy[j], q);
          float2 dd, v;
          dd.x = __fsub_rn(h.x, __shfl_up_sync(0xffffffffu, h.y, 1));
          dd.y = __fsub_rn(h.y, h.x);
#pragma unroll
          for (int e = 0; e < 2; ++e) el(v, e) = __fmul_rn(el(dd, e), el(ik, e));
          if (XS) {
            float2 p = lds(oX + (4 * j + 2 + q) * sX);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              el(p, e) = next(el(xb, e), el(p, e), el(xa, e), el(dd, e));
              el(v, e) = __fadd_rn(el(v, e), el(p, e));
            }
            sts(oX + (4 * j + 2 + q) * sX, p);
          }
          part(dx, q) = v;
        }
        // CA f + CB d
        auto update = [&](cf2& f, const float2* C, const cf2& d, int e) {
          const float fr = el(f.r, e), fi = el(f.i, e), ar = el(C[0], e), ai = el(C[1], e), br = el(C[2], e), bi = el(C[3], e);
          const float dr = el(d.r, e), di = el(d.i, e);
          el(f.r, e) = __fmaf_rn(ar, fr, __fmaf_rn(-ai, fi, __fmaf_rn(br, dr, -__fmul_rn(bi, di))));
          el(f.i, e) = __fmaf_rn(ar, fi, __fmaf_rn(ai, fr, __fmaf_rn(br, di, __fmul_rn(bi, dr))));
        };
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = i0 + e;
          if (CS || (i <= NX - 2 && k >= 1 && k <= NZ - 2)) update(ex[j], c, dz, e);
          if (CS || (i >= 1 && i <= NX - 2 && k <= NZ - 2)) update(ez[j], c + 4, dx, e);
        }
      }
      if (src >= 0) {  // :581-582
        const float* f = s0.io.src + a.t0 + s;
        const int n = s0.io.nstep;
#pragma unroll
        for (int q = 0; q < 2 * RB; ++q)
          if (q == src) {
            if (src_x) {
              el(ex[q / 2].r, q & 1) += f[0];
              el(ex[q / 2].i, q & 1) += f[n];
            }
            if (src_z) {
              el(ez[q / 2].r, q & 1) += f[2 * n];
              el(ez[q / 2].i, q & 1) += f[3 * n];
            }
          }
      }
      if (EDGE && !CS) {
#pragma unroll
        for (int j = 0; j < RB; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (x_plane(i0 + e, kb + j)) el(ex[j].r, e) = el(ex[j].i, e) = 0.0f;
            if (z_plane(i0 + e, kb + j)) el(ez[j].r, e) = el(ez[j].i, e) = 0.0f;
          }
      }
      if (EDGE && hyz) zero_hy();
      if (own) {  // the norm monitor of the owned cells (Ex up to NX - 2, Ez up to row NZ - 2)
        auto owned = [&](auto&& fn) {
#pragma unroll
          for (int j = 0; j < RB; ++j)
            if (own >> j & 1u)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const bool x = !XS || i0 + e <= NX - 2, z = !EDGE || (kb + j <= NZ - 2 && (!XS || i0 + e < NX));
                fn(x ? el(ex[j].r, e) : 0.0f, x ? el(ex[j].i, e) : 0.0f, z ? el(ez[j].r, e) : 0.0f,
                   z ? el(ez[j].i, e) : 0.0f);
              }
        };
        float big = 0.0f;
        owned([&](float xr, float xi, float zr, float zi) {
          big = max_nan(big, fabsf(xr) + fabsf(xi) + fabsf(zr) + fabsf(zi));
        });
        if (big <= 1e24f) {
          nrm = fmaxf(nrm, big);
        } else {  // near the threshold, or NaN: the norm itself
          float q4 = 0.0f;
          owned([&](float xr, float xi, float zr, float zi) { q4 = max_nan(q4, c2_norm4(xr, xi, zr, zi)); });
          nrm = fmaxf(nrm, nan_to_inf(sqrtf(sqrtf(q4)) * 1.2676506e30f));  // 2^100
        }
      }
      if (rec0 >= 0) {  // receivers of step t
        float* tr = s0.io.traces + (size_t)(a.t0 + s) * 4 * s0.io.nrec;
        const int n = s0.io.nrec;
        auto sample = [&](int r, int c) {  // cell c = 2 * row + element
          float v[4] = {0.f, 0.f, 0.f, 0.f};
          const unsigned cell = 1u << c;  // a bit, or the compiler indexes the fields in local memory
#pragma unroll
          for (int u = 0; u < 2 * RB; ++u) {
            const bool at = cell >> u & 1u;
            v[0] = at ? el(ex[u / 2].r, u & 1) : v[0];
            v[1] = at ? el(ex[u / 2].i, u & 1) : v[1];
            v[2] = at ? el(ez[u / 2].r, u & 1) : v[2];
            v[3] = at ? el(ez[u / 2].i, u & 1) : v[3];
          }
#pragma unroll
          for (int m = 0; m < 4; ++m) tr[(size_t)m * n + r] = v[m];
        };
#pragma unroll 1
        for (int q = rec0, next; q >= 0; q = next) {
          int r = q, c;
          if (listed) {
            next = G.next[q];
            r = G.rec[q] >> 4;
            c = G.rec[q] & 15;
          } else {
            next = q + 1 < n ? q + 1 : -1;
            const int e = s0.io.rec[3 * q] - i0, j = s0.io.rec[3 * q + 2] - kb;
            if (e < 0 || e > 1 || j < 0 || j >= RB || !(own >> j & 1u)) continue;
            c = 2 * j + e;
          }
          sample(r, c);
        }
      }
      show_e();
    }
    __syncthreads();
  }

  // ---- write the owned cells; what no loop updates is carried over
  if (own) {
    float* const zm[4] = {a.mExz[0], a.mExz[1], a.mHyz[0], a.mHyz[1]};
    float* const xm[4] = {a.mEzx[0], a.mEzx[1], a.mHyx[0], a.mHyx[1]};
    const float* const zf[4] = {s0.mExz[0], s0.mExz[1], s0.mHyz[0], s0.mHyz[1]};
    const float* const xf[4] = {s0.mEzx[0], s0.mEzx[1], s0.mHyx[0], s0.mHyx[1]};
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      if (!(own >> j & 1u)) continue;
      const size_t g = (size_t)k * P + i0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        *reinterpret_cast<float2*>(a.Ex[q] + g) = part(ex[j], q);
        *reinterpret_cast<float2*>(a.Ez[q] + g) = part(ez[j], q);
        float2 h = part(hy[j], q);
        if (EDGE && k > NZ - 2)  // no loop advances row NZ - 1
#pragma unroll
          for (int e = 0; e < 2; ++e)
            el(h, e) = i0 + e == 0 || i0 + e == NX - 2 ? 0.0f : s0.Hy[q][g + e];
        *reinterpret_cast<float2*>(a.Hy[q] + g) = h;
      }
      if (EDGE && in_strip(k, NZ, W)) {
        const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float2 p = lds(oZ(k) + q * kCC);
          if (XS && i0 + 1 > NX - 2)  // nor column NX - 1
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if (i0 + e > NX - 2) el(p, e) = zf[q][zg + e];
          *reinterpret_cast<float2*>(zm[q] + zg) = p;
        }
      }
      if (xsl) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = i0 + e;
          if (i >= NX || !in_strip(i, NX, W)) continue;
          const size_t xg = (size_t)k * (2 * W) + strip_idx(i, NX, W);
#pragma unroll
          for (int q = 0; q < 4; ++q) xm[q][xg] = k > NZ - 2 ? xf[q][xg] : c2_smem[oX + (4 * j + q) * sX + e];
        }
      }
    }
  }
  block_norm_to_slot(nrm, s0.io.slots, blockIdx.x);
}

template <int RB>
__global__ void __launch_bounds__(kThreads, 1)
    em2c_stream_kernel(const __grid_constant__ Em2cStream a, int ntx, int nbz, int smem) {
  __shared__ C2Tile G;
  const int NX = a.from.NX, NZ = a.from.NZ, W = a.from.W;
  const C2Frame f = c2_frame(NX, NZ, W, RB, ntx, nbz, blockIdx.x % ntx, blockIdx.x / ntx);
  const bool xs = f.bx < W || f.xend > NX - W;
  const bool edge = xs || f.bx < 1 || f.xend > NX - 2 || f.bz < max(W, 1) || f.kend > NZ - max(W, 2);
  if (4 * f.end > smem) em2c_tile<RB, true, true, false>(a, G, f);
  else if (!edge) em2c_tile<RB, false, false, true>(a, G, f);
  else if (!xs) em2c_tile<RB, true, false, true>(a, G, f);
  else em2c_tile<RB, true, true, true>(a, G, f);
}

using Kernel = void (*)(Em2cStream, int, int, int);
const Kernel kKernels[kMaxRows] = {em2c_stream_kernel<1>, em2c_stream_kernel<2>, em2c_stream_kernel<3>,
                                   em2c_stream_kernel<4>, em2c_stream_kernel<5>};

}  // namespace

cudaError_t em2c_stream_prepare(int NX, int NZ, int W, StreamPlan* out) {
  int dev = 0, sms = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  const int limit = optin - (int)sizeof(C2Tile) - 256;  // the kernels' static shared memory (and block_norm_to_slot's)
  const int ng = (NX + 1) / 2, most = (kCC - 2 * kC2Halo) / 2;
  out->ntx = NX <= kCC ? 1 : (ng + most - 1) / most;
  double best = 1e30;
  for (int rb = 1; rb <= kMaxRows; ++rb) {  // the rows a warp whose waves of tiles take least
    const int F = kWarps * rb, nbz = NZ <= F ? 1 : (NZ + F - 2 * kC2Halo - 1) / (F - 2 * kC2Halo);
    const double cost = ((out->ntx * nbz + sms - 1) / sms) * (kC2TileCost + rb);
    if (cost > best) continue;
    best = cost;
    out->rb = rb;
    out->nbz = nbz;
  }
  int need = 0;
  for (int r = 0; r < out->nbz; ++r)
    for (int c = 0; c < out->ntx; ++c) {
      const C2Frame f = c2_frame(NX, NZ, W, out->rb, out->ntx, out->nbz, c, r);
      need = std::max(need, 4 * f.end <= limit ? 4 * f.end : 4 * f.oC);
    }
  out->smem = need;
  return res_allow_max_smem((const void*)kKernels[out->rb - 1]);
}

void em2c_stream_launch(const Em2cStream& a, const StreamPlan& plan, cudaStream_t s) {
  kKernels[plan.rb - 1]<<<plan.ntx * plan.nbz, kThreads, plan.smem, s>>>(a, plan.ntx, plan.nbz, (int)plan.smem);
}

}  // namespace sfd

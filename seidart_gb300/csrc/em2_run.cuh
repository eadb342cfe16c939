// The electromag2 tile's run: loading the frame, the steps, the hand-over
// between the tiles of an on-chip run (resident2d.cu) and the write-back; the
// streaming steps (em2_stream.cu) share all but the hand-over.  Internal
// linkage: each translation unit that includes it gets its own copy.
#pragma once
#include <type_traits>

#include "em2_tile.cuh"

namespace sfd {

using namespace res;
using namespace tile2;

namespace {

// Place of cell i of row k among the hand-over words: the cells e of every
// lane's four lie together, so that a warp's store of one of them writes 512
// consecutive bytes.
__device__ __forceinline__ size_t em2_word(int k, int i, int P) { return (size_t)k * P + (i & 3) * (P >> 2) + (i >> 2); }

// Elements 0 .. n - 1 of v, zero from there on.
__device__ __forceinline__ float4 em2_below(float4 v, int n) {
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (e >= n) el(v, e) = 0.0f;
  return v;
}

extern __shared__ __align__(16) float em2_smem[];

// A tile's geometry and the places of its arrays in em2_smem (in floats), in
// shared memory: what a hand-over or the end of the run needs of it is read
// there instead of being held in registers through the steps.
struct Em2Tile {
  int ox0, ox1, oz0, oz1;      // owned cells
  int bx, bz, xend, kend;      // frame
  int wlo, wh0;                // warps below wlo and from wh0 on hold a row that rounds dEz/dx (em2_rounded_z)
  int xlo, xh0, nxl;           // lanes below xlo and from xh0 on hold an x-strip cell; their number
  int zn;                      // frame rows in a z strip
  int hS;                      // floats of a field of the halo
  unsigned tag;                // of the last hand-over
  int nrec, nmine, abort;      // receivers: of the tile, of the threads counted so far; a wait gave up
  int oZ, oX, oH;              // z and x memory variables, halo
  int nget, npub;              // entries of the lists of the hand-over
  int oGet, oPub;              // and their places
  int rec[2 * kResMaxLocalRec];  // (receiver, frame cell) pairs
  int mine[kResMaxLocalRec];     // the same, each thread's together: receiver << 4 | 4 * row + element
};

// One CTA's tile, owning columns te.x .. te.y - 1 and rows te.z .. te.w - 1, for
// a.nsteps steps.  MODE 0: a run on chip; 1: a recompute for the adjoint (every
// step's state dumped, the handle's state kept); 2: a run that also saves
// checkpoints; kStream: at most kTileHalo steps from one copy of the state to
// the other, with no hand-over.  EDGE: the frame holds CPML strip or boundary
// cells.  XS: it holds x-strip cells or columns that round dEz/dx (em2_rounded_x).
//
// Nothing updates Hy in row NZ - 1 and column NX - 1 or the memory variables
// there (:249-295), and no update reads them: the registers' values are left
// to run there, and the stored ones stay as they are in global memory.
//
// em2_smem: [6][128] x tables ik ad b ikh adh bh, [warps][128] first Ex row of
// each warp, [warps][128] last Hy row of each warp, [4 warps][8] row tables ik b
// ad - ikh bh adh -, [R][4][128] CAx CBx CAz CBz (RB > kEm2KeepRows), the rows of
// the warps with a z-strip row [][2][128] (dEx_dz, dHy_dz; zero tables in the
// rows outside the strip), the x-strip lanes [R][2][nxl][4] (dEz_dx, dHy_dx),
// and for the hand-over Ex, Ez, Hy of the halo.  What a step reads lies at places known to the compiler: a place read from shared
// memory first would put two round trips in the chain of a half-step.
#ifndef EM2_RUN_WARPS
#define EM2_RUN_WARPS kEm2MaxWarps  // most warps of the including file's CTAs
#endif
constexpr int kOEx = 6 * kCols, kOHy = kOEx + EM2_RUN_WARPS * kCols, kORT = kOHy + EM2_RUN_WARPS * kCols,
              kOC = kORT + 8 * 4 * EM2_RUN_WARPS;
constexpr int kStream = 3;  // em2_run_tile's mode of a few steps from copy to copy
// Words a thread has in flight in a hand-over.
constexpr int kBatch = 3;
// Most entries of the lists of a hand-over (em2_run_tile): of a tile with
// hrows halo rows, hown owned rows, zrows frame rows in a z strip, xlanes lanes
// with x-strip cells.
__host__ __device__ constexpr int em2_get_entries(int hrows, int hown, int zrows, int xlanes) {
  return (hrows + (hrows < zrows ? hrows : zrows)) * kCols + 8 * (hown + (hown < zrows ? hown : zrows)) +
         4 * xlanes * hrows + (xlanes ? 8 * hown : 0);
}
__host__ __device__ constexpr int em2_pub_entries(int hown, int zrows, int xlanes) {
  return (2 * kTileHalo < zrows ? 2 * kTileHalo : zrows) * kCols + 8 * (hown < zrows ? hown : zrows) +
         4 * xlanes * 2 * kTileHalo + (xlanes ? 8 * hown : 0);
}
// Up to this many rows a warp the coefficients stay in registers.
constexpr int kEm2KeepRows = 1;

template <int RB, int MODE, bool EDGE, bool XS>
__device__ __forceinline__ void em2_run_tile(const Em2Resident& a, Em2Tile& G, int4 te) {
  constexpr bool DUMP = MODE == 1, CKPT = MODE == 2, STREAM = MODE == kStream, KEEP = RB <= kEm2KeepRows, KEEPT = RB <= 2;
  constexpr int kRow = 4 * kCols;  // floats from a row's coefficients to the next row's
  const int NX = a.NX, NZ = a.NZ, P = a.P, W = a.W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  Ctl* const ctl = a.io.ctl;
  const bool up = te.z > 0, down = te.w < NZ, left = te.x > 0, right = te.y < NX;
  const bool neighbours = !STREAM && (up || down || left || right);
  // the first receiver a thread looks at, on its way while the frame is loaded
  const int rec_i = tid < a.io.nrec ? __ldg(a.io.rec + 3 * tid) : -1, rec_k = tid < a.io.nrec ? __ldg(a.io.rec + 3 * tid + 2) : 0;
  const int bx = left ? te.x - kTileHalo : 0, bz = max(te.z - kTileHalo, 0);
  const int xend = min(NX, te.y + kTileHalo), kend = min(NZ, te.w + kTileHalo);
  const int R = (kend - bz + RB - 1) / RB * RB;
  const int nr = min(max(kend - bz - warp * RB, 0), RB);  // frame rows of this warp
  const int oC = kOC + warp * RB * kRow + 4 * lane;        // + j kRow + q kCols
  const int oRT = kORT + 8 * warp * RB;

  // ---- load the frame: every load of the fields and the coefficients is on
  // its way before anything waits
  float4 ex[RB], ez[RB], hy[RB], keep[KEEP ? RB : 1][4];
  unsigned own = 0, hyz = 0;  // owned rows of this lane; cells (bit 4 * row + element) where Hy is a Dirichlet plane
  int src = -1;               // 4 * row + element of the source cell
  {
    const int i0 = bx + 4 * lane, kb = bz + warp * RB;
    const bool lact = i0 < xend, lown = i0 >= te.x && i0 < te.y;
    const float* const coef[4] = {a.CAx, a.CBx, a.CAz, a.CBz};
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      const bool on = j < nr && lact;
      const size_t g = on ? (size_t)k * P + i0 : 0;
      if (!KEEP && warp * RB + j < R) {
#pragma unroll
        for (int q = 0; q < 4; ++q) copy16(em2_smem + oC + j * kRow + q * kCols, coef[q] + g, on);
      }
      if (KEEP)
#pragma unroll
        for (int q = 0; q < 4; ++q) keep[KEEP ? j : 0][q] = on ? ld4(coef[q] + g) : zero4;
      ex[j] = on ? *reinterpret_cast<const float4*>(a.Ex + g) : zero4;
      ez[j] = on ? *reinterpret_cast<const float4*>(a.Ez + g) : zero4;
      hy[j] = on ? *reinterpret_cast<const float4*>(a.Hy + g) : zero4;
      if (on && k == a.io.sk && a.io.si >= i0 && a.io.si < i0 + 4) src = 4 * j + a.io.si - i0;
      if (on && lown && k >= te.z && k < te.w) own |= 1u << j;
    }
  }
  if (tid == 0) {
    G.ox0 = te.x; G.ox1 = te.y; G.oz0 = te.z; G.oz1 = te.w;
    G.bx = bx; G.bz = bz; G.xend = xend; G.kend = kend;
    G.zn = max(min(W, kend) - bz, 0) + max(kend - max(NZ - W, bz), 0);
    G.wlo = (max(min(W, kend) - bz, 0) + RB - 1) / RB;
    G.wh0 = max((max(NZ - max(W, 2), bz) - bz) / RB, G.wlo);
    G.xlo = max((min(W, xend) - bx + 3) / 4, 0);
    G.xh0 = max((NX - W - bx) / 4, G.xlo);
    G.nxl = G.xlo + max((xend - bx + 3) / 4 - G.xh0, 0);
    G.oZ = kOC + (KEEP ? 0 : kRow * R);
    G.oX = G.oZ + (EDGE ? 2 * kCols * RB * (G.wlo + max(R / RB - G.wh0, 0)) : 0);
    G.oH = G.oX + (EDGE ? 8 * R * G.nxl : 0);
    const int hown = G.oz1 - G.oz0, hrows = G.oz0 - bz + kend - G.oz1;
    G.hS = hrows * kCols + 8 * hown;
    G.oGet = (G.oH + 3 * G.hS + 1) & ~1;
    G.oPub = G.oGet + 2 * em2_get_entries(hrows, hown, EDGE ? G.zn : 0, EDGE ? G.nxl : 0);
    G.nrec = G.nmine = G.nget = G.npub = G.abort = 0;
    // k_begin counted this run's hand-overs on
    if (!STREAM) G.tag = *(volatile unsigned*)&ctl->seq - (unsigned)em2_hand_overs(a.nsteps);
  }
  // rows past the frame are read as zero
  for (int q = tid; q < 2 * EM2_RUN_WARPS * kCols / 4; q += blockDim.x) sts4(em2_smem + kOEx + 4 * q, zero4);
  {
    const int i0 = bx + 4 * lane, kb = bz + warp * RB;
    const float* const xt[6] = {a.X.ik, a.X.ad, a.X.b, a.X.ikh, a.X.adh, a.X.bh};
    if (warp < 6) {  // the x tables, one a warp
      for (int q = warp; q < 6; q += min(6, (int)blockDim.x >> 5)) {
        float4 t = i0 < xend ? ld4(xt[q] + i0) : zero4;
        if (EDGE)
#pragma unroll
          for (int e = 0; e < 4; ++e) {  // memory variables outside the update loops stay zero
            if ((q == 1 || q == 2) && i0 + e > NX - 2) el(t, e) = 0.0f;
            if ((q == 4 || q == 5) && (i0 + e > NX - 2 || i0 + e < 1)) el(t, e) = 0.0f;
          }
        sts4(em2_smem + q * kCols + 4 * lane, t);
      }
    }
    // the row tables, lane 8 j + q entry q of row j
    const int j = lane >> 3, q = lane & 7, k = kb + j;
    if (j < RB && warp * RB + j < R) {
      const float* const zt[8] = {a.Z.ik, a.Z.b, a.Z.ad, nullptr, a.Z.ikh, a.Z.bh, a.Z.adh, nullptr};
      const bool on = j < nr && (q & 3) != 3 &&
                      ((q & 3) == 0 || (EDGE && in_strip(k, NZ, W) && k <= NZ - 2 && (q < 4 || k >= 1)));
      em2_smem[oRT + lane] = on ? __ldg(zt[q] + k) : 0.0f;
    }
  }
  __syncthreads();
  // this warp's rows, and whether this lane's columns, round dEz/dx (em2_rounded)
  unsigned rounded = 0;
  const bool roundx = XS && em2_rounded_x(bx + 4 * lane, NX, W);
  if (EDGE)
#pragma unroll
    for (int j = 0; j < RB; ++j)
      if (em2_rounded_z(bz + warp * RB + j, NZ, W)) rounded |= 1u << j;
  const unsigned roundall = roundx ? ~0u : rounded;
  constexpr bool xs = XS;                                                                  // the tile has x-strip lanes ...
  const bool xsl = xs && nr > 0 && bx + 4 * lane < xend && (lane < G.xlo || lane >= G.xh0);  // ... and this is one
  const bool zw = EDGE && nr > 0 && (warp < G.wlo || warp >= G.wh0);                       // this warp has a z-strip row
  const int oZ = G.oZ + 2 * kCols * RB * (warp < G.wlo ? warp : warp - G.wh0 + G.wlo) + 4 * lane;      // + (2 j + q) kCols
  const int sX = 4 * G.nxl, oX = G.oX + 2 * sX * RB * warp + 4 * (lane < G.xlo ? lane : lane - G.xh0 + G.xlo);  // + (2 j + q) sX
  if (EDGE) {
    const int i0 = bx + 4 * lane, kb = bz + warp * RB;
    const bool lact = i0 < xend;
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      if (warp * RB + j >= R) continue;
      const bool zs = in_strip(k, NZ, W);
      if (zw) {
        const bool on = j < nr && lact && zs;
        const size_t zg = (size_t)(on ? strip_idx(k, NZ, W) : 0) * P + i0;
        sts4(em2_smem + oZ + 2 * j * kCols, on ? *reinterpret_cast<const float4*>(a.mExz + zg) : zero4);
        sts4(em2_smem + oZ + (2 * j + 1) * kCols, on ? *reinterpret_cast<const float4*>(a.mHyz + zg) : zero4);
      }
      if (xsl) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = i0 + e;
          const bool on = j < nr && i < NX && in_strip(i, NX, W);
          const size_t xg = on ? (size_t)k * (2 * W) + strip_idx(i, NX, W) : 0;
          em2_smem[oX + 2 * j * sX + e] = on ? a.mEzx[xg] : 0.0f;
          em2_smem[oX + (2 * j + 1) * sX + e] = on ? a.mHyx[xg] : 0.0f;
        }
      }
    }
    if (!KEEP) copies_wait();
#pragma unroll
    for (int j = 0; j < RB; ++j) {  // loop bounds and planes into the coefficients
      const int k = kb + j;
      if (j >= nr || !lact || (k >= 1 && k <= NZ - 3 && i0 >= 1 && i0 + 3 <= NX - 3)) continue;
      float4 c[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) c[q] = KEEP ? keep[KEEP ? j : 0][q] : lds4(em2_smem + oC + j * kRow + q * kCols);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + e;
        if (i > NX - 2 || k < 1 || k > NZ - 2) {  // outside the Ex loop, :273-283
          el(c[0], e) = 1.0f;
          el(c[1], e) = 0.0f;
        }
        if (i > NX - 2 || i < 1 || k > NZ - 2) {  // outside the Ez loop, :285-295
          el(c[2], e) = 1.0f;
          el(c[3], e) = 0.0f;
        }
        if (i == 0 || i == NX - 2 || i >= NX || k == 0 || k == NZ - 1) el(c[0], e) = el(c[1], e) = 0.0f;  // planes,
        if (i == 0 || i >= NX - 1 || k == 0 || k == NZ - 2) el(c[2], e) = el(c[3], e) = 0.0f;             // :304-312
        if (k <= NZ - 2 && i <= NX - 2 && (i == 0 || i == NX - 2 || k == 0 || k == NZ - 2)) hyz |= 1u << (4 * j + e);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (KEEP) keep[KEEP ? j : 0][q] = c[q];
        else sts4(em2_smem + oC + j * kRow + q * kCols, c[q]);
      }
    }
  }
  // ---- receivers of the owned cells: listed by tile, then by thread (a tile
  // with more than it can list scans the whole list every step instead)
  for (int q = tid; q < a.io.nrec; q += blockDim.x) {
    const int i = q == tid ? rec_i : a.io.rec[3 * q], k = q == tid ? rec_k : a.io.rec[3 * q + 2];
    if (i >= G.ox0 && i < G.ox1 && k >= G.oz0 && k < G.oz1) {
      const int pos = atomicAdd(&G.nrec, 1);
      if (pos < kResMaxLocalRec) {
        G.rec[2 * pos] = q;
        G.rec[2 * pos + 1] = ((k - G.bz) << 7) | (i - G.bx);
      }
    }
  }
  if (nr > 0) sts4(em2_smem + kOEx + warp * kCols + 4 * lane, ex[0]);
  __syncthreads();
  int r0 = 0, r1 = 0;  // this thread's entries of G.mine; r1 = -1: scan
  {
    const int n = G.nrec;
    if (n <= kResMaxLocalRec) {
      auto mine = [&](int q) {
        const int c = G.rec[2 * q + 1], row = (c >> 7) - warp * RB, col = (c & 127) - 4 * lane;
        return row >= 0 && row < RB && col >= 0 && col < 4 ? 4 * row + col : -1;
      };
      int m = 0;
      for (int q = 0; q < n; ++q) m += mine(q) >= 0;
      if (m > 0) {
        r0 = r1 = atomicAdd(&G.nmine, m);
        for (int q = 0; q < n; ++q)
          if (mine(q) >= 0) G.mine[r1++] = G.rec[2 * q] << 4 | mine(q);
      }
    } else if (own) {
      r1 = -1;
    }
  }

  // ---- the hand-over (see the file comment).  Its code runs once in
  // kTileHalo steps, when none of it is in the instruction caches, so it is
  // kept short: what it moves is listed once per run.  Entries: the word's
  // place, and the place in em2_smem with the kind -- 0 a halo cell's field
  // word (three floats, G.hS apart), 1 a z-strip word (two, kCols apart), 2 an
  // x-strip word (two, sX apart).  get: every word of the halo; pub: the
  // strips' words of the owned cells that lie in a neighbour's halo (their
  // fields come from registers).
  int2* const get = reinterpret_cast<int2*>(em2_smem + G.oGet);
  int2* const pub = reinterpret_cast<int2*>(em2_smem + G.oPub);
  const int wz = NZ * P, wx = wz + 2 * W * P;  // places of the first z- and x-strip words
  const size_t words = (size_t)wx + (size_t)NZ * 2 * W;
  unsigned ring = 0;  // owned rows of this lane that lie in a neighbour's halo
  if (neighbours) {
    const int htop = G.oz0 - G.bz, hown = G.oz1 - G.oz0, ncols = (G.xend - G.bx + 3) & ~3;
    const int nB = (htop + G.kend - G.oz1) * kCols;
    auto strips = [&](int2* list, int* count, int r, int c) {  // the strip words of frame cell (r, c)
      const int k = G.bz + r, i = G.bx + c;
      if (EDGE && in_strip(k, NZ, W)) {
        const int w = r / RB, row = (w < G.wlo ? w : w - G.wh0 + G.wlo) * RB + r % RB;
        list[atomicAdd(count, 1)] =
            make_int2(wz + (int)em2_word(strip_idx(k, NZ, W), i, P), (G.oZ + 2 * kCols * row + c) | 1 << 28);
      }
      if (XS && i < NX && in_strip(i, NX, W)) {
        const int l = c >> 2, at = G.oX + 2 * r * sX + 4 * (l < G.xlo ? l : l - G.xh0 + G.xlo) + (c & 3);
        list[atomicAdd(count, 1)] = make_int2(wx + k * 2 * W + strip_idx(i, NX, W), at | 2 << 28);
      }
    };
    const int nL = nB + (left ? 4 * hown : 0), nH = nL + (right ? 4 * hown : 0);
    for (int q = tid; q < nH; q += blockDim.x) {  // the fields first, row by row in the words' order
      const bool lf = q < nL;
      const int m = q - (lf ? nB : nL), h = q >> 7;
      const int r = q < nB ? (h < htop ? h : h + hown) : htop + (m >> 2);
      const int c = q < nB ? ((q & 31) << 2) | ((q >> 5) & 3) : (lf ? 0 : ncols - 4) + (m & 3);
      const int slot = q < nB ? h * kCols + c : nB + 8 * (m >> 2) + (lf ? 0 : 4) + (m & 3);
      get[q] = c < ncols ? make_int2((int)em2_word(G.bz + r, G.bx + c, P), G.oH + slot) : make_int2(-1, 0);
    }
    if (tid == 0) G.nget = nH;
    __syncthreads();
    if (EDGE) {
      for (int q = tid; q < nH; q += blockDim.x) {
        const bool lf = q < nL;
        const int m = q - (lf ? nB : nL), h = q >> 7;
        const int r = q < nB ? (h < htop ? h : h + hown) : htop + (m >> 2);
        const int c = q < nB ? q & 127 : (lf ? 0 : ncols - 4) + (m & 3);
        if (c < ncols) strips(get, &G.nget, r, c);
      }
    }
    const int i0 = G.bx + 4 * lane;
    const bool lring = (left && i0 == G.ox0) || (right && i0 == G.ox1 - kTileHalo);
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int r = warp * RB + j, k = G.bz + r;
      if ((own >> j & 1u) && (lring || (up && k < G.oz0 + kTileHalo) || (down && k >= G.oz1 - kTileHalo))) {
        ring |= 1u << j;
        if (EDGE)
          for (int e = 0; e < 4; ++e) strips(pub, &G.npub, r, 4 * lane + e);
      }
    }
    __syncthreads();
  }
  auto hand_over = [&] {  // every thread of the CTA
    const unsigned tag = G.tag + 1u, want = tag + a.tag_bias;
    uint4* const word = a.words + (tag & 1u) * words;
    uint4* const mine = word + em2_word(G.bz + warp * RB, G.bx + 4 * lane, P);
#pragma unroll
    for (int j = 0; j < RB; ++j)
      if (ring >> j & 1u)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          st_word(mine + j * P + e * (P >> 2), el(ex[j], e), el(ez[j], e), el(hy[j], e), tag);
    if (EDGE) {
      __syncthreads();  // every warp's memory variables are there, and their halo's places are done with
#pragma unroll 1
      for (int q = tid; q < G.npub; q += blockDim.x) {
        const int2 t = pub[q];
        const float* p = em2_smem + (t.y & 0xfffffff);
        st_word(word + t.x, p[0], p[t.y >> 28 == 1 ? kCols : sX], 0.0f, tag);
      }
    }
    unsigned long long t0 = 0;
    const int n = G.nget;
#pragma unroll 1
    for (int q0 = tid; q0 < n; q0 += kBatch * blockDim.x) {
      int2 t[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int q = q0 + u * (int)blockDim.x;
        t[u] = q < n ? get[q] : make_int2(-1, 0);
      }
#pragma unroll 1
      for (int it = 1;; ++it) {
        uint4 v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (t[u].x >= 0) v[u] = ld_word(word + t[u].x);
        bool more = false;
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          if (t[u].x < 0) continue;
          if (v[u].w != want) {
            more = true;
            continue;
          }
          const int kind = EDGE ? t[u].y >> 28 : 0;
          float* p = em2_smem + (t[u].y & 0xfffffff);
          p[0] = __uint_as_float(v[u].x);
          p[kind == 0 ? G.hS : kind == 1 ? kCols : sX] = __uint_as_float(v[u].y);
          if (kind == 0) p[2 * G.hS] = __uint_as_float(v[u].z);
          t[u].x = -1;
        }
        if (!more) break;
        if ((it & 15) == 0 && !poll_again(ctl, a.limit_ns, t0)) {
          G.abort = 1;
          break;
        }
      }
    }
    __syncthreads();
    if (tid == 0) G.tag = tag;
    // this thread's halo cells
    const int htop = G.oz0 - G.bz, hown = G.oz1 - G.oz0, i0 = G.bx + 4 * lane;
    if (i0 < G.xend) {
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const int r = warp * RB + j;
        if (j >= nr || (own >> j & 1u)) continue;
        const float* p = em2_smem + G.oH +
                         (r < htop           ? r * kCols + 4 * lane
                          : r >= htop + hown ? (r - hown) * kCols + 4 * lane
                                             : G.hS - 8 * (htop + hown - r) + (i0 < G.ox0 ? 0 : 4));
        ex[j] = lds4(p);
        ez[j] = lds4(p + G.hS);
        hy[j] = lds4(p + 2 * G.hS);
      }
    }
  };

  float4 tab[KEEPT ? 6 : 1];  // the x tables of this lane
  if (KEEPT)
#pragma unroll
    for (int q = 0; q < (KEEPT ? 6 : 1); ++q)
      if (xs || q % 3 == 0) tab[q] = lds4(em2_smem + q * kCols + 4 * lane);
  // H half-step of this warp's rows (electromagfdtd.f95:249-262).  ZS: with
  // the z strip's memory variables
  auto h_rows = [&](auto zs_tag) {
    constexpr bool ZS = decltype(zs_tag)::value;
    const float* T = em2_smem + 4 * lane;
    const float4 exb = lds4(em2_smem + kOEx + min(warp + 1, EM2_RUN_WARPS - 1) * kCols + 4 * lane);
    const float4 ik = KEEPT ? tab[0] : lds4(T);
    float4 xa, xb;
    if (xs) {
      xa = KEEPT ? tab[1] : lds4(T + kCols);
      xb = KEEPT ? tab[2] : lds4(T + 2 * kCols);
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
        const float4 exn = j < RB - 1 ? ex[j < RB - 1 ? j + 1 : j] : exb;
        const float ezn = __shfl_down_sync(0xffffffffu, ez[j].x, 1);
        const float4 rt = ZS ? lds4(em2_smem + oRT + 8 * j) : make_float4(em2_smem[oRT + 8 * j], 0.f, 0.f, 0.f);
        float4 dEx, dEz, v;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          el(dEx, e) = __fsub_rn(el(exn, e), el(ex[j], e));
          el(v, e) = __fmul_rn(el(dEx, e), rt.x);
        }
        if (ZS) {
          float4 p = lds4(em2_smem + oZ + 2 * j * kCols);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(p, e) = __fmaf_rn(rt.z, el(dEx, e), __fmul_rn(rt.y, el(p, e)));
            el(v, e) = __fadd_rn(el(v, e), el(p, e));
          }
          sts4(em2_smem + oZ + 2 * j * kCols, p);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          el(dEz, e) = __fsub_rn(e < 3 ? el(ez[j], e + 1) : ezn, el(ez[j], e));
        }
        float4 p = zero4;
        if (xs) {
          if (xsl) p = lds4(em2_smem + oX + 2 * j * sX);
#pragma unroll
          for (int e = 0; e < 4; ++e) el(p, e) = __fmaf_rn(el(xb, e), el(p, e), __fmul_rn(el(xa, e), el(dEz, e)));
          if (xsl) sts4(em2_smem + oX + 2 * j * sX, p);
        }
        // dEz/dx, rounded or fused into the sum (em2_rounded; where it is fused, p is
        // zero).  A select: two forms of the loop, or a branch a row, cost 4 to 7 %
        // of a step of 1040 x 540 cells, this 1 to 3 %; the mask alone costs frames of two
        // and four rows a warp 1 to 4 % more, the other way those of one and three.
        const bool round = RB & 1 ? roundall >> j & 1u : roundx || (rounded >> j & 1u);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float fused = __fmaf_rn(el(dEz, e), el(ik, e), el(v, e));
          float t = __fmul_rn(el(dEz, e), el(ik, e));
          if (xs) t = __fadd_rn(t, el(p, e));
          el(v, e) = (ZS || xs) && round ? __fadd_rn(t, el(v, e)) : fused;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) el(hy[j], e) = __fmaf_rn(a.dbH, el(v, e), el(hy[j], e));
    }
    sts4(em2_smem + kOHy + warp * kCols + 4 * lane, hy[RB - 1]);
  };
  // E half-step of this warp's rows (:273-295)
  auto e_rows = [&](auto zs_tag) {
    constexpr bool ZS = decltype(zs_tag)::value;
    const float* T = em2_smem + 3 * kCols + 4 * lane;
    const float4 hmt = lds4(em2_smem + kOHy + max(warp - 1, 0) * kCols + 4 * lane);
    const float4 ik = KEEPT ? tab[3] : lds4(T);
    float4 xa, xb;
    if (xs) {
      xa = KEEPT ? tab[4] : lds4(T + kCols);
      xb = KEEPT ? tab[5] : lds4(T + 2 * kCols);
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
        const float4 hm = j > 0 ? hy[j > 0 ? j - 1 : 0] : hmt;
        const float hl = __shfl_up_sync(0xffffffffu, hy[j].w, 1);
        const float4 rt = ZS ? lds4(em2_smem + oRT + 8 * j + 4) : make_float4(em2_smem[oRT + 8 * j + 4], 0.f, 0.f, 0.f);
        const float* C = em2_smem + oC + j * kRow;
        float4 dH, d;
        {
          const float4 ca = KEEP ? keep[KEEP ? j : 0][0] : lds4(C), cb = KEEP ? keep[KEEP ? j : 0][1] : lds4(C + kCols);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(dH, e) = __fsub_rn(el(hy[j], e), el(hm, e));
            el(d, e) = __fmul_rn(el(dH, e), rt.x);
          }
          if (ZS) {
            float4 p = lds4(em2_smem + oZ + (2 * j + 1) * kCols);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              el(p, e) = __fmaf_rn(rt.z, el(dH, e), __fmul_rn(rt.y, el(p, e)));
              el(d, e) = __fadd_rn(el(d, e), el(p, e));
            }
            sts4(em2_smem + oZ + (2 * j + 1) * kCols, p);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) el(ex[j], e) = __fmaf_rn(el(ca, e), el(ex[j], e), __fmul_rn(el(cb, e), el(d, e)));
        }
        const float4 ca = KEEP ? keep[KEEP ? j : 0][2] : lds4(C + 2 * kCols);
        const float4 cb = KEEP ? keep[KEEP ? j : 0][3] : lds4(C + 3 * kCols);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          el(dH, e) = __fsub_rn(el(hy[j], e), e == 0 ? hl : el(hy[j], e > 0 ? e - 1 : 0));
          el(d, e) = __fmul_rn(el(dH, e), el(ik, e));
        }
        if (xs) {
          float4 p = zero4;
          if (xsl) p = lds4(em2_smem + oX + (2 * j + 1) * sX);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(p, e) = __fmaf_rn(el(xb, e), el(p, e), __fmul_rn(el(xa, e), el(dH, e)));
            el(d, e) = __fadd_rn(el(d, e), el(p, e));
          }
          if (xsl) sts4(em2_smem + oX + (2 * j + 1) * sX, p);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) el(ez[j], e) = __fmaf_rn(el(ca, e), el(ez[j], e), __fmul_rn(el(cb, e), el(d, e)));
    }
  };
  // Hy of row j (grid row k) with the cells no loop updates as they are stored
  auto hy_stored = [&](int j, int k, int i0) {
    float4 v = hy[j];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (k > NZ - 2 || i0 + e > NX - 2) el(v, e) = a.Hy[(size_t)k * P + i0 + e];
    return v;
  };
  // the strip cells' memory variables at (j, e) of one of the arrays; zero at i = NX - 1, which no loop updates
  auto zpsi = [&](int j, int q, int i0) { return em2_below(lds4(em2_smem + oZ + (2 * j + q) * kCols), NX - 1 - i0); };

  if (!EDGE && !KEEP) copies_wait();  // each thread reads only what it copied
  float nrm = 0.0f;
  const bool rare = src >= 0 || hyz || r0 != r1;
  for (int s = 0; s < a.nsteps; ++s) {
    // a run with no hand-over in it has one before it, so that no tile writes
    // back what a neighbour has yet to load
    if (neighbours && (s > 0 ? s % kTileHalo == 0 : a.nsteps <= kTileHalo)) {
      hand_over();
      if (G.abort) return;  // the state is left as it was loaded; the host reports the timeout
      if (nr > 0) sts4(em2_smem + kOEx + warp * kCols + 4 * lane, ex[0]);
      __syncthreads();
    }
    if (zw) h_rows(std::true_type{});
    else if (nr > 0) h_rows(std::false_type{});
    __syncthreads();

    if (zw) e_rows(std::true_type{});
    else if (nr > 0) e_rows(std::false_type{});
    if (src >= 0) {  // :300-301
      const float fx = a.io.src[a.t0 + s], fz = a.io.src[a.io.nstep + a.t0 + s];
#pragma unroll
      for (int q = 0; q < 4 * RB; ++q)
        if (q == src) {
          el(ex[q / 4], q & 3) += fx;
          el(ez[q / 4], q & 3) += fz;
        }
    }
    if (own) {  // the norm monitor: |Ex| + |Ez| of the owned cells
      float big = 0.0f;
      if (own == (1u << RB) - 1u) {
#pragma unroll
        for (int j = 0; j < RB; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) big = max_nan(big, fabsf(el(ex[j], e)) + fabsf(el(ez[j], e)));
      } else {
#pragma unroll
        for (int j = 0; j < RB; ++j)
          if (own >> j & 1u)
#pragma unroll
            for (int e = 0; e < 4; ++e) big = max_nan(big, fabsf(el(ex[j], e)) + fabsf(el(ez[j], e)));
      }
      if (big <= 1e24f) {
        nrm = fmaxf(nrm, big);
      } else {  // near the threshold, or NaN: the 2-norm itself
        float sq = 0.0f;
#pragma unroll
        for (int j = 0; j < RB; ++j)
          if (own >> j & 1u)
#pragma unroll
            for (int e = 0; e < 4; ++e) sq = max_nan(sq, norm_sq(el(ex[j], e), el(ez[j], e)));
        nrm = fmaxf(nrm, norm_of_sq(sq));
      }
    }
    if (DUMP && own) {  // the state after step t; Hy before its planes are zeroed
      char* d = a.dump.base + (size_t)(s + 1) * a.dump.stride;
      const int i0 = G.bx + 4 * lane, kb = G.bz + warp * RB;
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const int k = kb + j;
        if (!(own >> j & 1u)) continue;
        const size_t g = (size_t)k * P + i0;
        // streaming stores: the copies are read back only after the run
        __stcs(reinterpret_cast<float4*>((float*)(d + a.dump.off[0]) + g), ex[j]);
        __stcs(reinterpret_cast<float4*>((float*)(d + a.dump.off[1]) + g), ez[j]);
        __stcs(reinterpret_cast<float4*>((float*)(d + a.dump.off[2]) + g),
               !EDGE || (k <= NZ - 2 && i0 + 3 <= NX - 2) ? hy[j] : hy_stored(j, k, i0));
        if (EDGE && in_strip(k, NZ, W)) {
          const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i0;
          __stcs(reinterpret_cast<float4*>((float*)(d + a.dump.off[3]) + zg), zpsi(j, 0, i0));
          __stcs(reinterpret_cast<float4*>((float*)(d + a.dump.off[5]) + zg), zpsi(j, 1, i0));
        }
        if (xsl) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (i0 + e < NX && in_strip(i0 + e, NX, W)) {
              const size_t xg = (size_t)k * (2 * W) + strip_idx(i0 + e, NX, W);
              ((float*)(d + a.dump.off[4]))[xg] = k <= NZ - 2 ? em2_smem[oX + 2 * j * sX + e] : a.mEzx[xg];
              ((float*)(d + a.dump.off[6]))[xg] = k <= NZ - 2 ? em2_smem[oX + (2 * j + 1) * sX + e] : a.mHyx[xg];
            }
        }
      }
    }
    if (rare) {
      if (EDGE && hyz) {  // the stored Hy keeps its Dirichlet planes at zero, after every row's E used it (:314-317)
#pragma unroll
        for (int q = 0; q < 4 * RB; ++q)
          if (hyz >> q & 1u) el(hy[q / 4], q & 3) = 0.0f;
      }
      if (r0 != r1) {  // receivers of step t
        float* tr = a.io.traces + (size_t)(a.t0 + s) * 2 * a.io.nrec;
        auto sample = [&](int r, int c) {  // cell c = 4 * row + element
          float vx = 0.0f, vz = 0.0f;
#pragma unroll
          for (int q = 0; q < 4 * RB; ++q)
            if (q == c) {
              vx = el(ex[q / 4], q & 3);
              vz = el(ez[q / 4], q & 3);
            }
          tr[r] = vx;
          tr[a.io.nrec + r] = vz;
        };
        if (r1 >= 0) {
          for (int q = r0; q < r1; ++q) sample(G.mine[q] >> 4, G.mine[q] & 15);
        } else {
          const int i0 = G.bx + 4 * lane, kb = G.bz + warp * RB;
          for (int q = 0; q < a.io.nrec; ++q) {
            const int e = a.io.rec[3 * q] - i0, j = a.io.rec[3 * q + 2] - kb;
            if (e >= 0 && e < 4 && j >= 0 && j < RB && (own >> j & 1u)) sample(q, 4 * j + e);
          }
        }
      }
    }
    if (CKPT && own && (s + 1) % a.ckpt_every == 0 && s + 1 < a.nsteps) {
      // a checkpoint: the state the handle would hold after step t, in the
      // sfd_checkpoint_save layout (scalar stores: the caller's rows need
      // only 4-byte alignment)
      char* d = a.ckpt.base + (size_t)((s + 1) / a.ckpt_every) * a.ckpt.stride;
      const int i0 = G.bx + 4 * lane, kb = G.bz + warp * RB;
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const int k = kb + j;
        if (!(own >> j & 1u)) continue;
        const size_t g = (size_t)k * P + i0;
        const bool zs = EDGE && in_strip(k, NZ, W);
        const float4 p = zs ? zpsi(j, 0, i0) : zero4, q = zs ? zpsi(j, 1, i0) : zero4;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = i0 + e;
          if (i >= NX) continue;
          __stcs((float*)(d + a.ckpt.off[0]) + g + e, el(ex[j], e));
          __stcs((float*)(d + a.ckpt.off[1]) + g + e, el(ez[j], e));
          __stcs((float*)(d + a.ckpt.off[2]) + g + e, i == NX - 1 || k == NZ - 1 ? a.Hy[g + e] : el(hy[j], e));
          if (zs) {
            const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i;
            __stcs((float*)(d + a.ckpt.off[3]) + zg, el(p, e));
            __stcs((float*)(d + a.ckpt.off[5]) + zg, el(q, e));
          }
          if (EDGE && in_strip(i, NX, W)) {
            const size_t xg = (size_t)k * (2 * W) + strip_idx(i, NX, W);
            __stcs((float*)(d + a.ckpt.off[4]) + xg, k <= NZ - 2 ? em2_smem[oX + 2 * j * sX + e] : a.mEzx[xg]);
            __stcs((float*)(d + a.ckpt.off[6]) + xg, k <= NZ - 2 ? em2_smem[oX + (2 * j + 1) * sX + e] : a.mHyx[xg]);
          }
        }
      }
    }
    if (nr > 0) sts4(em2_smem + kOEx + warp * kCols + 4 * lane, ex[0]);
    __syncthreads();
  }

  // ---- write the owned cells back (a recompute run for the adjoint keeps its input)
  if (!DUMP && own) {
    const int i0 = G.bx + 4 * lane, kb = G.bz + warp * RB;
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      if (!(own >> j & 1u)) continue;
      const size_t g = (size_t)k * P + i0;
      st4(a.oEx + g, ex[j]);
      st4(a.oEz + g, ez[j]);
      st4(a.oHy + g, !EDGE || (k <= NZ - 2 && i0 + 3 <= NX - 2) ? hy[j] : hy_stored(j, k, i0));
      if (EDGE && in_strip(k, NZ, W)) {
        const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i0;
        st4(a.omExz + zg, zpsi(j, 0, i0));
        st4(a.omHyz + zg, zpsi(j, 1, i0));
      }
      if (xsl && k <= NZ - 2) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (i0 + e < NX && in_strip(i0 + e, NX, W)) {
            const size_t xg = (size_t)k * (2 * W) + strip_idx(i0 + e, NX, W);
            a.omEzx[xg] = em2_smem[oX + 2 * j * sX + e];
            a.omHyx[xg] = em2_smem[oX + (2 * j + 1) * sX + e];
          }
      }
    }
  }
  block_norm_to_slot(nrm, a.io.slots, blockIdx.x);
}

}  // namespace
}  // namespace sfd

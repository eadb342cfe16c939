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
// takes 1.81 us (1.3 us of it the step of the largest tiles, the rest a
// hand-over of 2.2 us in four); 120 x 90 cells take 1.3 us.  The form before
// it exchanged one-cell edges twice a step, every cell mask applied in the
// step: 4.24 and 4.3 us.
//
// The per-cell arithmetic is that of the loops of
// legacy/fortran/electromagfdtd.f95:249-321.  Every product and sum names its
// rounding, so that a cell gets the same bits from whichever tile computes it
// (its own or one whose halo it lies in) and whichever form of the kernel: a
// run in pieces, with checkpoints or recomputed for the adjoint gives the
// states of the plain run.
#include <algorithm>
#include <type_traits>

#include "em2_tile.cuh"
#include "tile_plan.h"

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
  int wlo, wh0;                // warps below wlo and from wh0 on hold a z-strip row
  int xlo, xh0, nxl;           // lanes below xlo and from xh0 on hold an x-strip cell; their number
  int R, zn;                   // frame rows rounded up to whole warps, those of a z strip
  int hS;                      // floats of a field of the halo
  unsigned tag;                // of the last hand-over
  int nrec, nmine, abort;      // receivers: of the tile, of the threads counted so far; a wait gave up
  int oZ, oX, oH;              // z and x memory variables, halo
  int nget, npub;              // entries of the lists of the hand-over
  int oGet, oPub;              // and their places
  int rec[2 * kResMaxLocalRec];  // (receiver, frame cell) pairs
  int mine[kResMaxLocalRec];     // the same, each thread's together: receiver << 4 | 4 * row + element
};

// One CTA's tile for the whole run.  MODE 0: a run; 1: a recompute for the
// adjoint (every step's state dumped, the handle's state kept); 2: a run that
// also saves checkpoints.  EDGE: the frame holds CPML strip or boundary cells.
//
// Nothing updates Hy in row NZ - 1 and column NX - 1 or the memory variables
// there (:249-295), and no update reads them: the registers' values are left
// to run there, and the stored ones stay as they are in global memory.
//
// em2_smem: [6][128] x tables ik ad b ikh adh bh, [16][128] first Ex row of
// each warp, [16][128] last Hy row of each warp, [64][8] row tables ik b ad -
// ikh bh adh -, [R][4][128] CAx CBx CAz CBz (RB > kEm2KeepRows), the rows of
// the warps with a z-strip row [][2][128] (dEx_dz, dHy_dz; zero tables in the
// rows outside the strip), the x-strip lanes [R][2][nxl][4] (dEz_dx, dHy_dx),
// and for the hand-over Ex, Ez, Hy of the halo.  What a step reads lies at places known to the compiler: a place read from shared
// memory first would put two round trips in the chain of a half-step.
constexpr int kOEx = 6 * kCols, kOHy = kOEx + 16 * kCols, kORT = kOHy + 16 * kCols, kOC = kORT + 8 * 64;
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
__device__ __forceinline__ void em2_run_tile(const Em2Resident& a, Em2Tile& G) {
  constexpr bool DUMP = MODE == 1, CKPT = MODE == 2, KEEP = RB <= kEm2KeepRows, KEEPT = RB <= 2;
  constexpr int kRow = 4 * kCols;  // floats from a row's coefficients to the next row's
  const int NX = a.NX, NZ = a.NZ, P = a.P, W = a.W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  Ctl* const ctl = a.io.ctl;
  const int4 te = a.plan.tile[blockIdx.x];
  const bool up = (te.y & 0xffff) > 0, down = (te.y >> 16) < NZ, left = (te.x & 0xffff) > 0, right = (te.x >> 16) < NX;
  const bool neighbours = up || down || left || right;
  if (tid == 0) {
    G.ox0 = te.x & 0xffff; G.ox1 = te.x >> 16; G.oz0 = te.y & 0xffff; G.oz1 = te.y >> 16;
    G.bx = left ? G.ox0 - kTileHalo : 0;
    G.bz = max(G.oz0 - kTileHalo, 0);
    G.xend = min(NX, G.ox1 + kTileHalo);
    G.kend = min(NZ, G.oz1 + kTileHalo);
    G.R = (G.kend - G.bz + RB - 1) / RB * RB;
    G.zn = max(min(W, G.kend) - G.bz, 0) + max(G.kend - max(NZ - W, G.bz), 0);
    G.wlo = (max(min(W, G.kend) - G.bz, 0) + RB - 1) / RB;
    G.wh0 = max((max(NZ - W, G.bz) - G.bz) / RB, G.wlo);
    G.xlo = max((min(W, G.xend) - G.bx + 3) / 4, 0);
    G.xh0 = max((NX - W - G.bx) / 4, G.xlo);
    G.nxl = G.xlo + max((G.xend - G.bx + 3) / 4 - G.xh0, 0);
    G.oZ = kOC + (KEEP ? 0 : kRow * G.R);
    G.oX = G.oZ + (EDGE ? 2 * kCols * RB * (G.wlo + max(G.R / RB - G.wh0, 0)) : 0);
    G.oH = G.oX + (EDGE ? 8 * G.R * G.nxl : 0);
    const int hown = G.oz1 - G.oz0, hrows = G.oz0 - G.bz + G.kend - G.oz1;
    G.hS = hrows * kCols + 8 * hown;
    G.oGet = (G.oH + 3 * G.hS + 1) & ~1;
    G.oPub = G.oGet + 2 * em2_get_entries(hrows, hown, EDGE ? G.zn : 0, EDGE ? G.nxl : 0);
    G.nrec = G.nmine = G.nget = G.npub = G.abort = 0;
    // k_begin counted this run's hand-overs on
    G.tag = *(volatile unsigned*)&ctl->seq - (unsigned)em2_hand_overs(a.nsteps);
  }
  for (int q = tid; q < 32 * kCols; q += blockDim.x) em2_smem[kOEx + q] = 0.0f;  // rows past the frame are read as zero
  __syncthreads();
  const int nr = min(max(G.kend - G.bz - warp * RB, 0), RB);     // frame rows of this warp
  const int oC = kOC + warp * RB * kRow + 4 * lane;  // + j kRow + q kCols
  const int oRT = kORT + 8 * warp * RB;
  constexpr bool xs = XS;                                                                  // the tile has x-strip lanes ...
  const bool xsl = xs && nr > 0 && G.bx + 4 * lane < G.xend && (lane < G.xlo || lane >= G.xh0);      // ... and this is one
  const bool zw = EDGE && nr > 0 && (warp < G.wlo || warp >= G.wh0);                       // this warp has a z-strip row
  const int oZ = G.oZ + 2 * kCols * RB * (warp < G.wlo ? warp : warp - G.wh0 + G.wlo) + 4 * lane;      // + (2 j + q) kCols
  const int sX = 4 * G.nxl, oX = G.oX + 2 * sX * RB * warp + 4 * (lane < G.xlo ? lane : lane - G.xh0 + G.xlo);  // + (2 j + q) sX

  // ---- load the frame
  float4 ex[RB], ez[RB], hy[RB], keep[KEEP ? RB : 1][4];
  unsigned own = 0, hyz = 0;  // owned rows of this lane; cells (bit 4 * row + element) where Hy is a Dirichlet plane
  int src = -1;               // 4 * row + element of the source cell
  {
    const int i0 = G.bx + 4 * lane, kb = G.bz + warp * RB;
    const bool lact = i0 < G.xend, lown = i0 >= G.ox0 && i0 < G.ox1;
    if (warp == 0) {
      const float* tab[6] = {a.X.ik, a.X.ad, a.X.b, a.X.ikh, a.X.adh, a.X.bh};
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        float4 t = lact ? ld4(tab[q] + i0) : zero4;
        if (EDGE)
#pragma unroll
          for (int e = 0; e < 4; ++e) {  // memory variables outside the update loops stay zero
            if ((q == 1 || q == 2) && i0 + e > NX - 2) el(t, e) = 0.0f;
            if ((q == 4 || q == 5) && (i0 + e > NX - 2 || i0 + e < 1)) el(t, e) = 0.0f;
          }
        sts4(em2_smem + q * kCols + 4 * lane, t);
      }
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      ex[j] = ez[j] = hy[j] = zero4;
      if (KEEP)
#pragma unroll
        for (int q = 0; q < 4; ++q) keep[KEEP ? j : 0][q] = zero4;
      if (warp * RB + j >= G.R) continue;
      const bool zs = EDGE && in_strip(k, NZ, W);
      if (lane == 0) {
        float* rt = em2_smem + oRT + 8 * j;
        rt[0] = j < nr ? __ldg(a.Z.ik + k) : 0.0f;
        rt[4] = j < nr ? __ldg(a.Z.ikh + k) : 0.0f;
        const bool zh = j < nr && zs && k <= NZ - 2, ze = zh && k >= 1;
        rt[1] = zh ? __ldg(a.Z.b + k) : 0.0f;
        rt[2] = zh ? __ldg(a.Z.ad + k) : 0.0f;
        rt[5] = ze ? __ldg(a.Z.bh + k) : 0.0f;
        rt[6] = ze ? __ldg(a.Z.adh + k) : 0.0f;
      }
      float4 c[4] = {zero4, zero4, zero4, zero4};
      if (j < nr && lact) {
        const size_t g = (size_t)k * P + i0;
        ex[j] = *reinterpret_cast<const float4*>(a.Ex + g);
        ez[j] = *reinterpret_cast<const float4*>(a.Ez + g);
        hy[j] = *reinterpret_cast<const float4*>(a.Hy + g);
        c[0] = ld4(a.CAx + g);
        c[1] = ld4(a.CBx + g);
        c[2] = ld4(a.CAz + g);
        c[3] = ld4(a.CBz + g);
        if (EDGE) {
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
        }
        if (k == a.io.sk && a.io.si >= i0 && a.io.si < i0 + 4) src = 4 * j + a.io.si - i0;
        if (lown && k >= G.oz0 && k < G.oz1) own |= 1u << j;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (KEEP) keep[KEEP ? j : 0][q] = c[q];
        else sts4(em2_smem + oC + j * kRow + q * kCols, c[q]);
      }
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
  }
  // ---- receivers of the owned cells: listed by tile, then by thread (a tile
  // with more than it can list scans the whole list every step instead)
  for (int q = tid; q < a.io.nrec; q += blockDim.x) {
    const int i = a.io.rec[3 * q], k = a.io.rec[3 * q + 2];
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
    const float4 exb = lds4(em2_smem + kOEx + min(warp + 1, 15) * kCols + 4 * lane);
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
            el(p, e) = __fmaf_rn(rt.y, el(p, e), __fmul_rn(rt.z, el(dEx, e)));
            el(v, e) = __fadd_rn(el(v, e), el(p, e));
          }
          sts4(em2_smem + oZ + 2 * j * kCols, p);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          el(dEz, e) = __fsub_rn(e < 3 ? el(ez[j], e + 1) : ezn, el(ez[j], e));
          el(v, e) = __fmaf_rn(el(dEz, e), el(ik, e), el(v, e));
        }
        if (xs) {
          float4 p = zero4;
          if (xsl) p = lds4(em2_smem + oX + 2 * j * sX);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            el(p, e) = __fmaf_rn(el(xb, e), el(p, e), __fmul_rn(el(xa, e), el(dEz, e)));
            el(v, e) = __fadd_rn(el(v, e), el(p, e));
          }
          if (xsl) sts4(em2_smem + oX + 2 * j * sX, p);
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
              el(p, e) = __fmaf_rn(rt.y, el(p, e), __fmul_rn(rt.z, el(dH, e)));
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
      st4(a.Ex + g, ex[j]);
      st4(a.Ez + g, ez[j]);
      st4(a.Hy + g, !EDGE || (k <= NZ - 2 && i0 + 3 <= NX - 2) ? hy[j] : hy_stored(j, k, i0));
      if (EDGE && in_strip(k, NZ, W)) {
        const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i0;
        st4(a.mExz + zg, zpsi(j, 0, i0));
        st4(a.mHyz + zg, zpsi(j, 1, i0));
      }
      if (xsl && k <= NZ - 2) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (i0 + e < NX && in_strip(i0 + e, NX, W)) {
            const size_t xg = (size_t)k * (2 * W) + strip_idx(i0 + e, NX, W);
            a.mEzx[xg] = em2_smem[oX + 2 * j * sX + e];
            a.mHyx[xg] = em2_smem[oX + (2 * j + 1) * sX + e];
          }
      }
    }
  }
  block_norm_to_slot(nrm, a.io.slots, blockIdx.x);
}

template <int RB, int MODE>
__global__ void __launch_bounds__(32 * kEm2MaxWarps, 1) em2_resident_kernel(const __grid_constant__ Em2Resident a) {
  __shared__ Em2Tile G;
  const int kind = a.plan.tile[blockIdx.x].z;
  if (kind == 0) em2_run_tile<RB, MODE, false, false>(a, G);
  else if (kind == 1) em2_run_tile<RB, MODE, true, false>(a, G);
  else em2_run_tile<RB, MODE, true, true>(a, G);
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

// Shared memory of a frame with rb rows a warp, as em2_run_tile lays it out.
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

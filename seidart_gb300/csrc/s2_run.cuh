// The seismic2 tile's run (corrected physics): loading the frame, the steps, the
// hand-over between the tiles of an on-chip run (resident_s2.cu) and the
// write-back; the streaming steps (s2_stream.cu) share all but the hand-over.
// Internal linkage: each translation unit that includes it gets its own copy.
#pragma once
#include <type_traits>

#include "em2_tile.cuh"

namespace sfd {

using namespace res;
using tile2::copies_wait;
using tile2::copy8;
using tile2::ld_word;
using tile2::max_nan;
using tile2::norm_of_sq;
using tile2::norm_sq;
using tile2::poll_again;
using tile2::st_word;

namespace {

constexpr int kSC = 64;       // frame columns: 32 lanes x 2 cells
constexpr int kS2Warps = 16;  // most warps of a CTA
constexpr int kS2Keep = 1;    // up to this many rows a warp the coefficients stay in registers
constexpr int kS2Batch = 3;   // words a thread has in flight in a hand-over
// places in s2_smem (floats): x tables ik ad b ikh adh bh, each warp's first
// vx, first vz, last vx, last vz, each warp's first szz, last sxz, row tables
// [48][8] ik ikh - - b ad bh adh, coefficients [R][12][64]
constexpr int kSV = 6 * kSC, kSS = kSV + kS2Warps * 4 * kSC, kSRT = kSS + kS2Warps * 2 * kSC,
              kSCo = kSRT + 8 * kS2MaxRows * kS2Warps;

extern __shared__ __align__(16) float s2_smem[];

__device__ __forceinline__ float& el(float2& v, int e) { return (&v.x)[e]; }
__device__ __forceinline__ float el(const float2& v, int e) { return (&v.x)[e]; }
__device__ __forceinline__ float2 lds(int o) { return *reinterpret_cast<const float2*>(s2_smem + o); }
__device__ __forceinline__ void sts(int o, float2 v) { *reinterpret_cast<float2*>(s2_smem + o) = v; }

// Place of cell i's word w of row k among the hand-over words (a warp's store
// of one cell and word of every lane writes 512 consecutive bytes).
__device__ __forceinline__ int s2_word(int k, int w, int i, int P) {
  return ((2 * k + w) * 2 + (i & 1)) * (P >> 1) + (i >> 1);
}

// Most entries of the lists of a hand-over: of a tile with hrows halo rows, hown
// owned rows, zrows frame rows in a z strip, xlanes lanes with x-strip cells
// (two words a cell, fields and strips alike).
__host__ __device__ constexpr int s2_get_entries(int hrows, int hown, int zrows, int xlanes) {
  return 2 * ((hrows + (hrows < zrows ? hrows : zrows)) * kSC + 2 * kS2Halo * (hown + (hown < zrows ? hown : zrows)) +
              2 * xlanes * hrows + (xlanes ? 2 * kS2Halo * hown : 0));
}
__host__ __device__ constexpr int s2_pub_entries(int hown, int zrows, int xlanes) {
  return 2 * ((2 * kS2Halo < zrows ? 2 * kS2Halo : zrows) * kSC + 2 * kS2Halo * (hown < zrows ? hown : zrows) +
              2 * xlanes * 2 * kS2Halo + (xlanes ? 2 * kS2Halo * hown : 0));
}

// A tile's geometry and the places of its arrays, in shared memory (as Em2Tile).
struct S2Tile {
  int ox0, ox1, oz0, oz1, bx, bz, xend, kend;
  int wlo, wh0, xlo, xh0, nxl;  // warps and lanes with strip cells, as in Em2Tile
  int R, zn, hS;                // frame rows in whole warps, those of a z strip, floats of a field of the halo
  unsigned tag;
  int nrec, nmine, abort;
  int oZ, oX, oH, oGet, oPub, nget, npub;
  int rec[2 * kResMaxLocalRec], mine[kResMaxLocalRec];
};

// Memory variable q of the z strips' six and of the x strips' six, in
// sfd_num_memory's order, and whether cell (i, k) lies in the loop that
// advances it: 0, 1 the normal stresses', 2, 3 the shear stress's, 4, 5 the
// velocities'.
__device__ __forceinline__ constexpr int z_index(int q) { return q == 0 ? 1 : q == 1 ? 2 : q == 2 ? 9 : q == 3 ? 10 : q == 4 ? 5 : 7; }
__device__ __forceinline__ constexpr int x_index(int q) { return q == 0 ? 0 : q == 1 ? 3 : q == 2 ? 8 : q == 3 ? 11 : q == 4 ? 4 : 6; }
__device__ __forceinline__ bool in_loop(bool zstrip, int q, int i, int k, int NX, int NZ) {
  if (q < 2) return k >= 1 && i <= NX - 2;
  if (q < 4) return k <= NZ - 2 && i >= 1;
  return (q == 4) == zstrip ? k <= NZ - 2 && i <= NX - 2 : k >= 1 && i >= 1;  // szz_z, sxz_x: vz; sxz_z, sxx_x: vx
}

// One CTA's tile, owning columns te.x .. te.y - 1 and rows te.z .. te.w - 1, for
// a.nsteps steps.  MODE 0: a run on chip; 1: one that dumps every step's state and
// keeps the handle's; kS2Stream: at most kS2Steps steps from one copy of the state
// to the other, with no hand-over.
constexpr int kS2Stream = 3;
template <int RB, int MODE, bool EDGE, bool XS>
__device__ __forceinline__ void s2_run_tile(const Seis2Resident& a, S2Tile& G, int4 te) {
  constexpr bool DUMP = MODE == 1, STREAM = MODE == kS2Stream, KEEP = RB <= kS2Keep && !STREAM;
  constexpr int kRow = 12 * kSC;
  const int NX = a.NX, NZ = a.NZ, P = a.P, W = a.W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float2 zero2 = make_float2(0.f, 0.f);
  Ctl* const ctl = a.io.ctl;
  const bool up = te.z > 0, down = te.w < NZ, left = te.x > 0, right = te.y < NX;
  const bool neighbours = !STREAM && (up || down || left || right);
  float* const memory[12] = {a.m_vxx, a.m_vzz, a.m_vxz, a.m_vzx, a.m_sxx_x, a.m_szz_z,
                             a.m_sxz_x, a.m_sxz_z, a.m2_vxx, a.m2_vzz, a.m2_vxz, a.m2_vzx};
  if (tid == 0) {
    G.ox0 = te.x; G.ox1 = te.y; G.oz0 = te.z; G.oz1 = te.w;
    G.bx = left ? G.ox0 - kS2Halo : 0;
    G.bz = max(G.oz0 - kS2Halo, 0);
    G.xend = min(NX, G.ox1 + kS2Halo);
    G.kend = min(NZ, G.oz1 + kS2Halo);
    G.R = (G.kend - G.bz + RB - 1) / RB * RB;
    G.zn = max(min(W, G.kend) - G.bz, 0) + max(G.kend - max(NZ - W, G.bz), 0);
    G.wlo = (max(min(W, G.kend) - G.bz, 0) + RB - 1) / RB;
    G.wh0 = max((max(NZ - W, G.bz) - G.bz) / RB, G.wlo);
    G.xlo = max((min(W, G.xend) - G.bx + 1) / 2, 0);
    G.xh0 = max((NX - W - G.bx) / 2, G.xlo);
    G.nxl = G.xlo + max((G.xend - G.bx + 1) / 2 - G.xh0, 0);
    G.oZ = kSCo + (KEEP ? 0 : kRow * G.R);
    G.oX = G.oZ + (EDGE ? 6 * kSC * RB * (G.wlo + max(G.R / RB - G.wh0, 0)) : 0);
    G.oH = G.oX + (EDGE ? 12 * G.R * G.nxl : 0);
    const int hown = G.oz1 - G.oz0, hrows = G.oz0 - G.bz + G.kend - G.oz1;
    G.hS = hrows * kSC + 2 * kS2Halo * hown;
    G.oGet = (G.oH + 6 * G.hS + 1) & ~1;
    G.oPub = G.oGet + 2 * s2_get_entries(hrows, hown, EDGE ? G.zn : 0, EDGE ? G.nxl : 0);
    G.nrec = G.nmine = G.nget = G.npub = G.abort = 0;
    if (!STREAM) G.tag = *(volatile unsigned*)&ctl->seq - (unsigned)s2_hand_overs(a.nsteps);  // k_begin counted this run's on
  }
  for (int q = tid; q < kS2Warps * 6 * kSC; q += blockDim.x) s2_smem[kSV + q] = 0.0f;  // rows past the frame are read as zero
  __syncthreads();
  const int nr = min(max(G.kend - G.bz - warp * RB, 0), RB);  // frame rows of this warp
  const int oC = kSCo + warp * RB * kRow + 2 * lane, oRT = kSRT + 8 * warp * RB;
  const bool xsl = XS && nr > 0 && G.bx + 2 * lane < G.xend && (lane < G.xlo || lane >= G.xh0);
  const bool zw = EDGE && nr > 0 && (warp < G.wlo || warp >= G.wh0);
  const int oZ = G.oZ + 6 * kSC * RB * (warp < G.wlo ? warp : warp - G.wh0 + G.wlo) + 2 * lane;  // + (6 j + q) kSC
  const int sX = 2 * G.nxl;
  const int oX = G.oX + 6 * sX * RB * warp + 2 * (lane < G.xlo ? lane : lane - G.xh0 + G.xlo);  // + (6 j + q) sX

  // ---- load the frame
  float2 vx[RB], vz[RB], sxx[RB], szz[RB], sxz[RB], keep[KEEP ? RB : 1][12];
  unsigned own = 0, plane = 0;  // owned rows of this lane; cells (bit 2 * row + element) on a Dirichlet plane
  int src = -1;                 // 2 * row + element of the source cell
  if (STREAM) {  // every copy of a coefficient on its way before a field is waited for
    const int i0 = G.bx + 2 * lane, kb = G.bz + warp * RB;
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      if (warp * RB + j >= G.R) continue;
      const bool on = j < nr && i0 < G.xend;
      const size_t g = on ? (size_t)(kb + j) * P + i0 : 0;
#pragma unroll
      for (int q = 0; q < 12; ++q)
        if (q < 10 || a.atten) copy8(s2_smem + oC + j * kRow + q * kSC, a.coef[q] + g, on);
    }
  }
  {
    const int i0 = G.bx + 2 * lane, kb = G.bz + warp * RB;
    const bool lact = i0 < G.xend, lown = i0 >= G.ox0 && i0 < G.ox1;
    if (warp == 0) {
      const float* tab[6] = {a.X.ik, a.X.ad, a.X.b, a.X.ikh, a.X.adh, a.X.bh};
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        float2 t = lact ? *reinterpret_cast<const float2*>(tab[q] + i0) : zero2;
        if (EDGE && i0 + 1 >= NX) t.y = 0.0f;
        sts(q * kSC + 2 * lane, t);
      }
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      vx[j] = vz[j] = sxx[j] = szz[j] = sxz[j] = zero2;
      float2 c[12];
#pragma unroll
      for (int q = 0; q < 12; ++q) c[q] = zero2;
      if (warp * RB + j < G.R) {
        const bool zs = EDGE && j < nr && in_strip(k, NZ, W);
        if (lane == 0) {
          float* rt = s2_smem + oRT + 8 * j;
          rt[0] = j < nr ? __ldg(a.Z.ik + k) : 0.0f;
          rt[1] = j < nr ? __ldg(a.Z.ikh + k) : 0.0f;
          rt[4] = zs ? __ldg(a.Z.b + k) : 0.0f;
          rt[5] = zs ? __ldg(a.Z.ad + k) : 0.0f;
          rt[6] = zs ? __ldg(a.Z.bh + k) : 0.0f;
          rt[7] = zs ? __ldg(a.Z.adh + k) : 0.0f;
        }
        if (j < nr && lact) {
          const size_t g = (size_t)k * P + i0;
          vx[j] = *reinterpret_cast<const float2*>(a.vx + g);
          vz[j] = *reinterpret_cast<const float2*>(a.vz + g);
          sxx[j] = *reinterpret_cast<const float2*>(a.sxx + g);
          szz[j] = *reinterpret_cast<const float2*>(a.szz + g);
          sxz[j] = *reinterpret_cast<const float2*>(a.sxz + g);
#pragma unroll
          for (int q = 0; q < (STREAM ? 0 : 12); ++q) c[q] = *reinterpret_cast<const float2*>(a.coef[q] + g);
          if (EDGE) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int i = i0 + e;
              if (i < 1 || i > NX - 2 || k < 1 || k > NZ - 2) {  // a Dirichlet plane of vx and vz, :365-375
                el(c[8], e) = el(c[9], e) = 0.0f;
                plane |= 1u << (2 * j + e);
              }
            }
          }
          if (k == a.io.sk && a.io.si >= i0 && a.io.si < i0 + 2) src = 2 * j + a.io.si - i0;
          if (lown && k >= G.oz0 && k < G.oz1) own |= 1u << j;
        }
        if (!KEEP && !STREAM)
#pragma unroll
          for (int q = 0; q < 12; ++q) sts(oC + j * kRow + q * kSC, c[q]);
        if (zw) {
          const bool on = zs && lact;
          const size_t zg = (size_t)(on ? strip_idx(k, NZ, W) : 0) * P + i0;
#pragma unroll
          for (int q = 0; q < 6; ++q)
            sts(oZ + (6 * j + q) * kSC, on ? *reinterpret_cast<const float2*>(memory[z_index(q)] + zg) : zero2);
        }
        if (xsl) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const bool on = j < nr && i0 + e < NX && in_strip(i0 + e, NX, W);
            const size_t xg = on ? (size_t)k * (2 * W) + strip_idx(i0 + e, NX, W) : 0;
#pragma unroll
            for (int q = 0; q < 6; ++q) s2_smem[oX + (6 * j + q) * sX + e] = on ? memory[x_index(q)][xg] : 0.0f;
          }
        }
      }
      if (KEEP)
#pragma unroll
        for (int q = 0; q < 12; ++q) keep[KEEP ? j : 0][q] = c[q];
    }
  }
  if (STREAM) {
    copies_wait();  // each thread reads only what it copied
    if (EDGE && plane)  // c[8], c[9] of the Dirichlet planes, as above
#pragma unroll
      for (int q = 0; q < 2 * RB; ++q)
        if (plane >> q & 1u)
          s2_smem[oC + q / 2 * kRow + 8 * kSC + (q & 1)] = s2_smem[oC + q / 2 * kRow + 9 * kSC + (q & 1)] = 0.0f;
  }
  // ---- receivers of the owned cells: listed by tile, then by thread (a tile
  // with more than it can list scans the whole list every step instead)
  for (int q = tid; q < a.io.nrec; q += blockDim.x) {
    const int i = a.io.rec[3 * q], k = a.io.rec[3 * q + 2];
    if (i >= G.ox0 && i < G.ox1 && k >= G.oz0 && k < G.oz1) {
      const int pos = atomicAdd(&G.nrec, 1);
      if (pos < kResMaxLocalRec) {
        G.rec[2 * pos] = q;
        G.rec[2 * pos + 1] = ((k - G.bz) << 6) | (i - G.bx);
      }
    }
  }
  auto show_v = [&] {  // the velocities the next warps read
    const int o = kSV + warp * 4 * kSC + 2 * lane;
    sts(o, vx[0]);
    sts(o + kSC, vz[0]);
    sts(o + 2 * kSC, vx[RB - 1]);
    sts(o + 3 * kSC, vz[RB - 1]);
  };
  if (nr > 0) show_v();
  __syncthreads();
  int r0 = 0, r1 = 0;  // this thread's entries of G.mine; r1 = -1: scan
  {
    const int n = G.nrec;
    if (n <= kResMaxLocalRec) {
      auto mine = [&](int q) {
        const int c = G.rec[2 * q + 1], row = (c >> 6) - warp * RB, col = (c & 63) - 2 * lane;
        return row >= 0 && row < RB && col >= 0 && col < 2 ? 2 * row + col : -1;
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

  // ---- the hand-over: lists as in em2_run_tile, every entry three floats, a
  // stride apart that its kind tells -- 0 fields (G.hS), 1 z strip (kSC), 2 x
  // strip (sX)
  int2* const get = reinterpret_cast<int2*>(s2_smem + G.oGet);
  int2* const pub = reinterpret_cast<int2*>(s2_smem + G.oPub);
  const int wz = 2 * NZ * P, wx = wz + 2 * 2 * W * P;
  const size_t words = (size_t)wx + (size_t)NZ * 2 * 2 * W;
  unsigned ring = 0;  // owned rows of this lane that lie in a neighbour's halo
  if (neighbours) {
    const int htop = G.oz0 - G.bz, hown = G.oz1 - G.oz0, ncols = (G.xend - G.bx + 1) & ~1;
    const int nB = (htop + G.kend - G.oz1) * kSC;
    auto strips = [&](int2* list, int* count, int r, int c) {  // the strip words of frame cell (r, c)
      const int k = G.bz + r, i = G.bx + c;
      if (EDGE && in_strip(k, NZ, W)) {
        const int w = r / RB, row = (w < G.wlo ? w : w - G.wh0 + G.wlo) * RB + r % RB;
        for (int h = 0; h < 2; ++h)
          list[atomicAdd(count, 1)] =
              make_int2(wz + s2_word(strip_idx(k, NZ, W), h, i, P), (G.oZ + (6 * row + 3 * h) * kSC + c) | 1 << 28);
      }
      if (XS && i < NX && in_strip(i, NX, W)) {
        const int l = c >> 1, at = G.oX + 6 * r * sX + 2 * (l < G.xlo ? l : l - G.xh0 + G.xlo) + (c & 1);
        for (int h = 0; h < 2; ++h)
          list[atomicAdd(count, 1)] =
              make_int2(wx + (2 * k + h) * 2 * W + strip_idx(i, NX, W), (at + 3 * h * sX) | 2 << 28);
      }
    };
    const int nL = nB + (left ? kS2Halo * hown : 0), nH = nL + (right ? kS2Halo * hown : 0);
    for (int q = tid; q < nH; q += blockDim.x) {  // the fields first, row by row in the words' order
      const bool lf = q < nL;
      const int m = q - (lf ? nB : nL), h = q >> 6;
      const int r = q < nB ? (h < htop ? h : h + hown) : htop + m / kS2Halo;
      const int c = q < nB ? ((q & 31) << 1) | ((q >> 5) & 1) : (lf ? 0 : ncols - kS2Halo) + m % kS2Halo;
      const int slot = q < nB ? h * kSC + c : nB + 2 * kS2Halo * (m / kS2Halo) + (lf ? 0 : kS2Halo) + m % kS2Halo;
      for (int h2 = 0; h2 < 2; ++h2)
        get[h2 * nH + q] =
            c < ncols ? make_int2(s2_word(G.bz + r, h2, G.bx + c, P), G.oH + 3 * h2 * G.hS + slot) : make_int2(-1, 0);
    }
    if (tid == 0) G.nget = 2 * nH;
    __syncthreads();
    if (EDGE) {
      for (int q = tid; q < nH; q += blockDim.x) {
        const bool lf = q < nL;
        const int m = q - (lf ? nB : nL), h = q >> 6;
        const int r = q < nB ? (h < htop ? h : h + hown) : htop + m / kS2Halo;
        const int c = q < nB ? q & 63 : (lf ? 0 : ncols - kS2Halo) + m % kS2Halo;
        if (c < ncols) strips(get, &G.nget, r, c);
      }
    }
    const int i0 = G.bx + 2 * lane;
    const bool lring = (left && i0 < G.ox0 + kS2Halo) || (right && i0 >= G.ox1 - kS2Halo);
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int r = warp * RB + j, k = G.bz + r;
      if ((own >> j & 1u) && (lring || (up && k < G.oz0 + kS2Halo) || (down && k >= G.oz1 - kS2Halo))) {
        ring |= 1u << j;
        if (EDGE)
          for (int e = 0; e < 2; ++e) strips(pub, &G.npub, r, 2 * lane + e);
      }
    }
    __syncthreads();
  }
  auto hand_over = [&] {  // every thread of the CTA
    const unsigned tag = G.tag + 1u, want = tag + a.tag_bias;
    uint4* const word = a.words + (tag & 1u) * words;
    uint4* const mine = word + s2_word(G.bz + warp * RB, 0, G.bx + 2 * lane, P);
#pragma unroll
    for (int j = 0; j < RB; ++j)
      if (ring >> j & 1u)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint4* w = mine + 2 * j * P + e * (P >> 1);
          st_word(w, el(vx[j], e), el(vz[j], e), el(sxx[j], e), tag);
          st_word(w + P, el(szz[j], e), el(sxz[j], e), 0.0f, tag);
        }
    if (EDGE) {
      __syncthreads();  // every warp's memory variables are there, and their halo's places are done with
#pragma unroll 1
      for (int q = tid; q < G.npub; q += blockDim.x) {
        const int2 t = pub[q];
        const float* p = s2_smem + (t.y & 0xfffffff);
        const int st = t.y >> 28 == 1 ? kSC : sX;
        st_word(word + t.x, p[0], p[st], p[2 * st], tag);
      }
    }
    unsigned long long t0 = 0;
    const int n = G.nget;
#pragma unroll 1
    for (int q0 = tid; q0 < n; q0 += kS2Batch * blockDim.x) {
      int2 t[kS2Batch];
#pragma unroll
      for (int u = 0; u < kS2Batch; ++u) {
        const int q = q0 + u * (int)blockDim.x;
        t[u] = q < n ? get[q] : make_int2(-1, 0);
      }
#pragma unroll 1
      for (int it = 1;; ++it) {
        uint4 v[kS2Batch];
#pragma unroll
        for (int u = 0; u < kS2Batch; ++u)
          if (t[u].x >= 0) v[u] = ld_word(word + t[u].x);
        bool more = false;
#pragma unroll
        for (int u = 0; u < kS2Batch; ++u) {
          if (t[u].x < 0) continue;
          if (v[u].w != want) {
            more = true;
            continue;
          }
          const int kind = EDGE ? t[u].y >> 28 : 0, st = kind == 0 ? G.hS : kind == 1 ? kSC : sX;
          float* p = s2_smem + (t[u].y & 0xfffffff);
          p[0] = __uint_as_float(v[u].x);
          p[st] = __uint_as_float(v[u].y);
          p[2 * st] = __uint_as_float(v[u].z);
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
    const int htop = G.oz0 - G.bz, hown = G.oz1 - G.oz0, i0 = G.bx + 2 * lane, hS = G.hS;
    if (i0 < G.xend) {
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const int r = warp * RB + j;
        if (j >= nr || (own >> j & 1u)) continue;
        const int o = G.oH + (r < htop           ? r * kSC + 2 * lane
                              : r >= htop + hown ? (r - hown) * kSC + 2 * lane
                                                 : hS - 2 * kS2Halo * (htop + hown - r) +
                                                       (i0 < G.ox0 ? i0 - G.bx : kS2Halo + i0 - G.ox1));
        vx[j] = lds(o);
        vz[j] = lds(o + hS);
        sxx[j] = lds(o + 2 * hS);
        szz[j] = lds(o + 3 * hS);
        sxz[j] = lds(o + 4 * hS);
      }
    }
  };

  auto coef = [&](int j, int q) { return KEEP ? keep[KEEP ? j : 0][q] : lds(oC + j * kRow + q * kSC); };
  // b m + ad d: a memory variable's next value
  auto next = [](float b, float m, float ad, float d) { return __fmaf_rn(b, m, __fmul_rn(ad, d)); };
  float2 tab[KEEP ? 6 : 1];  // the x tables of this lane
  if (KEEP)
#pragma unroll
    for (int q = 0; q < (KEEP ? 6 : 1); ++q) tab[q] = lds(q * kSC + 2 * lane);
  auto table = [&](int q) { return KEEP ? tab[KEEP ? q : 0] : lds(q * kSC + 2 * lane); };

  // The stresses of this warp's rows (seismicfdtd.f95:247-312).  ZS: with the
  // z strip's memory variables (zero tables in the rows outside it)
  auto stress_rows = [&](auto zs_tag) {
    constexpr bool ZS = decltype(zs_tag)::value;
    const int oU = kSV + (max(warp - 1, 0) * 4 + 2) * kSC + 2 * lane, oD = kSV + min(warp + 1, kS2Warps - 1) * 4 * kSC + 2 * lane;
    const float2 vxt = lds(oU), vzt = lds(oU + kSC), vxb = lds(oD), vzb = lds(oD + kSC);
    const float2 ikx = table(0), ikxh = table(3);
    float2 adx, bx, adxh, bxh;
    if (XS) {
      adx = table(1);
      bx = table(2);
      adxh = table(4);
      bxh = table(5);
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const float2 vxu = j > 0 ? vx[j > 0 ? j - 1 : 0] : vxt, vzu = j > 0 ? vz[j > 0 ? j - 1 : 0] : vzt;
      const float2 vxd = j < RB - 1 ? vx[j < RB - 1 ? j + 1 : j] : vxb, vzd = j < RB - 1 ? vz[j < RB - 1 ? j + 1 : j] : vzb;
      const float vxl = __shfl_up_sync(0xffffffffu, vx[j].y, 1), vzl = __shfl_up_sync(0xffffffffu, vz[j].y, 1);
      const float vxr = __shfl_down_sync(0xffffffffu, vx[j].x, 1), vzr = __shfl_down_sync(0xffffffffu, vz[j].x, 1);
      const float2 rt = lds(oRT + 8 * j);  // ikz ikzh
      const float4 zt = ZS ? res::lds4(s2_smem + oRT + 8 * j + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      // the four differences of either loop: x+ of vx, vz and z- of vz, vx; x- and z+
      float2 dxx, dzx, dzz, dxz;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        el(dxx, e) = __fsub_rn(e == 0 ? vx[j].y : vxr, el(vx[j], e));
        el(dzx, e) = __fsub_rn(e == 0 ? vz[j].y : vzr, el(vz[j], e));
        el(dzz, e) = __fsub_rn(el(vz[j], e), el(vzu, e));
        el(dxz, e) = __fsub_rn(el(vx[j], e), el(vxu, e));
      }
      auto gradients = [&](int xm, int zm) {  // scaled, with memory variables xm, xm + 1 of the x strip, zm, zm + 1 of the z strip
        float2 mxx = zero2, mzx = zero2, mzz = zero2, mxz = zero2;
        if (XS) {
          if (xsl) {
            mxx = lds(oX + (6 * j + xm) * sX);
            mzx = lds(oX + (6 * j + xm + 1) * sX);
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            el(mxx, e) = next(el(bxh, e), el(mxx, e), el(adxh, e), el(dxx, e));
            el(mzx, e) = next(el(bx, e), el(mzx, e), el(adx, e), el(dzx, e));
          }
          if (xsl) {
            sts(oX + (6 * j + xm) * sX, mxx);
            sts(oX + (6 * j + xm + 1) * sX, mzx);
          }
        }
        if (ZS) {
          mzz = lds(oZ + (6 * j + zm) * kSC);
          mxz = lds(oZ + (6 * j + zm + 1) * kSC);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            el(mzz, e) = next(zt.x, el(mzz, e), zt.y, el(dzz, e));
            el(mxz, e) = next(zt.z, el(mxz, e), zt.w, el(dxz, e));
          }
          sts(oZ + (6 * j + zm) * kSC, mzz);
          sts(oZ + (6 * j + zm + 1) * kSC, mxz);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          el(dxx, e) = XS ? __fmaf_rn(el(dxx, e), el(ikxh, e), el(mxx, e)) : __fmul_rn(el(dxx, e), el(ikxh, e));
          el(dzx, e) = XS ? __fmaf_rn(el(dzx, e), el(ikx, e), el(mzx, e)) : __fmul_rn(el(dzx, e), el(ikx, e));
          el(dzz, e) = ZS ? __fmaf_rn(el(dzz, e), rt.x, el(mzz, e)) : __fmul_rn(el(dzz, e), rt.x);
          el(dxz, e) = ZS ? __fmaf_rn(el(dxz, e), rt.y, el(mxz, e)) : __fmul_rn(el(dxz, e), rt.y);
          el(dzx, e) = __fadd_rn(el(dzx, e), el(dxz, e));  // the shear
        }
      };
      gradients(0, 0);
      {
        const float2 A11 = coef(j, 0), A13 = coef(j, 1), A15 = coef(j, 2), A33 = coef(j, 3), A35 = coef(j, 4);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float t = __fmaf_rn(el(A15, e), el(dzx, e), __fmaf_rn(el(A11, e), el(dxx, e), __fmul_rn(el(A13, e), el(dzz, e))));
          const float u = __fmaf_rn(el(A35, e), el(dzx, e), __fmaf_rn(el(A13, e), el(dxx, e), __fmul_rn(el(A33, e), el(dzz, e))));
          el(sxx[j], e) = __fadd_rn(el(sxx[j], e), t);
          el(szz[j], e) = __fadd_rn(el(szz[j], e), u);
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        el(dxx, e) = __fsub_rn(el(vx[j], e), e == 0 ? vxl : vx[j].x);
        el(dzx, e) = __fsub_rn(el(vz[j], e), e == 0 ? vzl : vz[j].x);
        el(dzz, e) = __fsub_rn(el(vzd, e), el(vz[j], e));
        el(dxz, e) = __fsub_rn(el(vxd, e), el(vx[j], e));
      }
      gradients(2, 2);
      {
        const float2 B15 = coef(j, 5), B35 = coef(j, 6), B55 = coef(j, 7);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float t = __fmaf_rn(el(B55, e), el(dzx, e), __fmaf_rn(el(B15, e), el(dxx, e), __fmul_rn(el(B35, e), el(dzz, e))));
          el(sxz[j], e) = __fadd_rn(el(sxz[j], e), t);
        }
      }
    }
  };
  // The velocities of this warp's rows (:317-357).  Both derivatives are rounded
  // before they are added: next to a source they cancel, and a fused product
  // leaves the other's rounding error in the velocity every step.
  auto velocity_rows = [&](auto zs_tag) {
    constexpr bool ZS = decltype(zs_tag)::value;
    const float2 sxzt = lds(kSS + (max(warp - 1, 0) * 2 + 1) * kSC + 2 * lane);
    const float2 szzb = lds(kSS + min(warp + 1, kS2Warps - 1) * 2 * kSC + 2 * lane);
    const float2 ikx = table(0), ikxh = table(3);
    float2 adx, bx, adxh, bxh;
    if (XS) {
      adx = table(1);
      bx = table(2);
      adxh = table(4);
      bxh = table(5);
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const float2 sxzu = j > 0 ? sxz[j > 0 ? j - 1 : 0] : sxzt, szzd = j < RB - 1 ? szz[j < RB - 1 ? j + 1 : j] : szzb;
      const float sxxl = __shfl_up_sync(0xffffffffu, sxx[j].y, 1), sxzr = __shfl_down_sync(0xffffffffu, sxz[j].x, 1);
      const float2 rt = lds(oRT + 8 * j);  // ikz ikzh
      const float4 zt = ZS ? res::lds4(s2_smem + oRT + 8 * j + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      float2 d1, d2, e1, e2;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        el(d1, e) = __fsub_rn(el(sxx[j], e), e == 0 ? sxxl : sxx[j].x);
        el(d2, e) = __fsub_rn(el(sxz[j], e), el(sxzu, e));
        el(e1, e) = __fsub_rn(e == 0 ? sxz[j].y : sxzr, el(sxz[j], e));
        el(e2, e) = __fsub_rn(el(szzd, e), el(szz[j], e));
      }
      float2 m1 = zero2, n1 = zero2;
      if (XS) {
        if (xsl) {
          m1 = lds(oX + (6 * j + 4) * sX);
          n1 = lds(oX + (6 * j + 5) * sX);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          el(m1, e) = next(el(bx, e), el(m1, e), el(adx, e), el(d1, e));
          el(n1, e) = next(el(bxh, e), el(n1, e), el(adxh, e), el(e1, e));
        }
        if (xsl) {
          sts(oX + (6 * j + 4) * sX, m1);
          sts(oX + (6 * j + 5) * sX, n1);
        }
      }
      if (ZS) {
        float2 n2 = lds(oZ + (6 * j + 4) * kSC), m2 = lds(oZ + (6 * j + 5) * kSC);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          el(m2, e) = next(zt.x, el(m2, e), zt.y, el(d2, e));
          el(n2, e) = next(zt.z, el(n2, e), zt.w, el(e2, e));
        }
        sts(oZ + (6 * j + 4) * kSC, n2);
        sts(oZ + (6 * j + 5) * kSC, m2);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          el(d2, e) = __fadd_rn(__fmul_rn(el(d2, e), rt.x), el(m2, e));
          el(e2, e) = __fadd_rn(__fmul_rn(el(e2, e), rt.y), el(n2, e));
        }
      } else {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          el(d2, e) = __fmul_rn(el(d2, e), rt.x);
          el(e2, e) = __fmul_rn(el(e2, e), rt.y);
        }
      }
      const float2 rx = coef(j, 8), rz = coef(j, 9);
      if (a.atten) {
        const float2 gx = coef(j, 10), gz = coef(j, 11);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          el(vx[j], e) = __fmul_rn(el(vx[j], e), el(gx, e));
          el(vz[j], e) = __fmul_rn(el(vz[j], e), el(gz, e));
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float s = __fmul_rn(el(d1, e), el(ikx, e)), t = __fmul_rn(el(e1, e), el(ikxh, e));
        if (XS) {
          s = __fadd_rn(s, el(m1, e));
          t = __fadd_rn(t, el(n1, e));
        }
        el(vx[j], e) = __fmaf_rn(__fadd_rn(s, el(d2, e)), el(rx, e), el(vx[j], e));
        el(vz[j], e) = __fmaf_rn(__fadd_rn(t, el(e2, e)), el(rz, e), el(vz[j], e));
      }
    }
  };
  // add `v0`, `v1`, `v2` to the source cell of f0, f1, f2
  auto add_at_source = [&](float2* f0, float2* f1, float2* f2, const float* amp, int s) {
#pragma unroll
    for (int q = 0; q < 2 * RB; ++q)
      if (q == src) {
        el(f0[q / 2], q & 1) += amp[a.t0 + s];
        el(f1[q / 2], q & 1) += amp[a.io.nstep + a.t0 + s];
        if (f2) el(f2[q / 2], q & 1) += amp[2 * a.io.nstep + a.t0 + s];
      }
  };

  float nrm = 0.0f;
  const bool rare = src >= 0 || plane || r0 != r1;
  for (int s = 0; s < a.nsteps; ++s) {
    // a run with no hand-over in it has one before it, so that no tile writes
    // back what a neighbour has yet to load
    if (neighbours && (s > 0 ? s % kS2Steps == 0 : a.nsteps <= kS2Steps)) {
      hand_over();
      if (G.abort) return;  // the state is left as it was loaded; the host reports the timeout
      if (nr > 0) show_v();
      __syncthreads();
    }
    if (nr > 0) {
      if (zw) stress_rows(std::true_type{});
      else stress_rows(std::false_type{});
      if (src >= 0 && a.io.ssrc) add_at_source(sxx, szz, sxz, a.io.ssrc, s);  // sigma_ij += f_ij(t) dt
      sts(kSS + warp * 2 * kSC + 2 * lane, szz[0]);
      sts(kSS + (warp * 2 + 1) * kSC + 2 * lane, sxz[RB - 1]);
    }
    __syncthreads();
    if (nr > 0) {
      if (zw) velocity_rows(std::true_type{});
      else velocity_rows(std::false_type{});
      if (rare) {
        if (src >= 0) add_at_source(vx, vz, nullptr, a.io.src, s);  // :360-361
        if (EDGE && plane) {  // :365-375
#pragma unroll
          for (int q = 0; q < 2 * RB; ++q)
            if (plane >> q & 1u) el(vx[q / 2], q & 1) = el(vz[q / 2], q & 1) = 0.0f;
        }
        if (r0 != r1) {  // receivers of step t
          float* tr = a.io.traces + (size_t)(a.t0 + s) * 2 * a.io.nrec;
          auto sample = [&](int r, int c) {  // cell c = 2 * row + element
            float x = 0.0f, z = 0.0f;
#pragma unroll
            for (int q = 0; q < 2 * RB; ++q)
              if (q == c) {
                x = el(vx[q / 2], q & 1);
                z = el(vz[q / 2], q & 1);
              }
            tr[r] = x;
            tr[a.io.nrec + r] = z;
          };
          if (r1 >= 0) {
            for (int q = r0; q < r1; ++q) sample(G.mine[q] >> 4, G.mine[q] & 15);
          } else {
            const int i0 = G.bx + 2 * lane, kb = G.bz + warp * RB;
            for (int q = 0; q < a.io.nrec; ++q) {
              const int e = a.io.rec[3 * q] - i0, j = a.io.rec[3 * q + 2] - kb;
              if (e >= 0 && e < 2 && j >= 0 && j < RB && (own >> j & 1u)) sample(q, 2 * j + e);
            }
          }
        }
      }
      if (own) {  // the norm monitor: |vx| + |vz| of the owned cells
        float big = 0.0f;
#pragma unroll
        for (int j = 0; j < RB; ++j)
          if (own >> j & 1u)
#pragma unroll
            for (int e = 0; e < 2; ++e) big = max_nan(big, fabsf(el(vx[j], e)) + fabsf(el(vz[j], e)));
        if (big <= 1e24f) {
          nrm = fmaxf(nrm, big);
        } else {  // near the threshold, or NaN: the 2-norm itself
          float sq = 0.0f;
#pragma unroll
          for (int j = 0; j < RB; ++j)
            if (own >> j & 1u)
#pragma unroll
              for (int e = 0; e < 2; ++e) sq = max_nan(sq, norm_sq(el(vx[j], e), el(vz[j], e)));
          nrm = fmaxf(nrm, norm_of_sq(sq));
        }
      }
      if (DUMP && own) {  // the state after step t into slot s + 1 (streaming stores: read once, by the adjoint)
        char* slot = a.dump.base + a.dump.stride * (size_t)(s + 1);
        auto arr = [&](int q) { return reinterpret_cast<float*>(slot + a.dump.off[q]); };
        const int i0 = G.bx + 2 * lane, kb = G.bz + warp * RB;
#pragma unroll
        for (int j = 0; j < RB; ++j) {
          const int k = kb + j;
          if (!(own >> j & 1u)) continue;
          const size_t g = (size_t)k * P + i0;
          __stcs(reinterpret_cast<float2*>(arr(0) + g), vx[j]);
          __stcs(reinterpret_cast<float2*>(arr(1) + g), vz[j]);
          __stcs(reinterpret_cast<float2*>(arr(2) + g), sxx[j]);
          __stcs(reinterpret_cast<float2*>(arr(3) + g), szz[j]);
          __stcs(reinterpret_cast<float2*>(arr(4) + g), sxz[j]);
          if (EDGE && in_strip(k, NZ, W)) {
            const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i0;
#pragma unroll
            for (int q = 0; q < 6; ++q) {
              float2 m = lds(oZ + (6 * j + q) * kSC);
#pragma unroll
              for (int e = 0; e < 2; ++e)
                if (i0 + e >= NX || !in_loop(true, q, i0 + e, k, NX, NZ)) el(m, e) = 0.0f;
              __stcs(reinterpret_cast<float2*>(arr(5 + z_index(q)) + zg), m);
            }
          }
          if (xsl) {
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if (i0 + e < NX && in_strip(i0 + e, NX, W)) {
                const size_t xg = (size_t)k * (2 * W) + strip_idx(i0 + e, NX, W);
#pragma unroll
                for (int q = 0; q < 6; ++q)
                  __stcs(arr(5 + x_index(q)) + xg,
                         in_loop(false, q, i0 + e, k, NX, NZ) ? s2_smem[oX + (6 * j + q) * sX + e] : 0.0f);
              }
          }
        }
      }
      show_v();
    }
    __syncthreads();
  }

  // ---- write the owned cells back (a recompute for the adjoint keeps its input)
  if (!DUMP && own) {
    const int i0 = G.bx + 2 * lane, kb = G.bz + warp * RB;
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int k = kb + j;
      if (!(own >> j & 1u)) continue;
      const size_t g = (size_t)k * P + i0;
      float* const field[5] = {a.vx, a.vz, a.sxx, a.szz, a.sxz};
      const float2 v[5] = {vx[j], vz[j], sxx[j], szz[j], sxz[j]};
#pragma unroll
      for (int q = 0; q < 5; ++q) *reinterpret_cast<float2*>((STREAM ? a.out[q] : field[q]) + g) = v[q];
      if (EDGE && in_strip(k, NZ, W)) {
        const size_t zg = (size_t)strip_idx(k, NZ, W) * P + i0;
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const bool in = i0 + e < NX && in_loop(true, q, i0 + e, k, NX, NZ);
            float* const m = STREAM ? a.out[5 + z_index(q)] : memory[z_index(q)];
            if (in) m[zg + e] = s2_smem[oZ + (6 * j + q) * kSC + e];
            else if (STREAM) m[zg + e] = memory[z_index(q)][zg + e];
          }
      }
      if (xsl) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (i0 + e < NX && in_strip(i0 + e, NX, W)) {
            const size_t xg = (size_t)k * (2 * W) + strip_idx(i0 + e, NX, W);
#pragma unroll
            for (int q = 0; q < 6; ++q) {
              float* const m = STREAM ? a.out[5 + x_index(q)] : memory[x_index(q)];
              if (in_loop(false, q, i0 + e, k, NX, NZ)) m[xg] = s2_smem[oX + (6 * j + q) * sX + e];
              else if (STREAM) m[xg] = memory[x_index(q)][xg];
            }
          }
      }
    }
  }
  block_norm_to_slot(nrm, a.io.slots, blockIdx.x);
}

}  // namespace
}  // namespace sfd

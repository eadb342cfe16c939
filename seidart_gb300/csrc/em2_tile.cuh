// The electromag2 tile: the cells one CTA advances by itself, several steps
// at a time, and the halo that lets it.
//
// A tile owns a rectangle of cells and works on a frame of it, the rectangle
// and kTileHalo cells more on every side that has a neighbour.  An electromag2
// step moves information by one cell (Hy reads Ex, Ez one cell up the axes;
// Ex, Ez read Hy one cell down), so after kTileHalo steps the owned cells are
// still what a step over the whole grid gives, while the halo's values are
// used up and are taken from the neighbours again: one hand-over between
// tiles for kTileHalo steps instead of two a step.  The halo's recomputation
// costs 128 x 42 cells of frame for 120 x 34 owned ones.
//
// A warp holds RB whole frame rows of 128 columns, four cells a lane, Ex, Ez
// and Hy in registers.  The neighbours along x are then in the same warp (one
// shuffle a row and half-step), those along z in the same thread but for the
// first and the last row of a warp, which pass through one row of shared
// memory each.  Every thread's coefficients and memory variables lie in
// shared memory in its own 16-byte slots, so no access conflicts.  The rows
// of a z strip are whole warps' rows: the strip recursion is a uniform
// branch.  The Fortran's loop bounds and Dirichlet planes of Ex and Ez
// (electromagfdtd.f95:273-312) are coefficient values -- (1, 0) carries a cell
// over, (0, 0) holds it at zero -- set when the tile is loaded.
#pragma once
#include "resident_common.cuh"

namespace sfd {
namespace tile2 {
namespace {

using res::lds2;
using res::lds4;
using res::sts4;

constexpr int kCols = 128;  // frame columns: 32 lanes x 4 cells

// A hand-over word: three values and the tag of the hand-over they belong
// to, written and read as one 128-bit access.
__device__ __forceinline__ uint4 ld_word(const uint4* p) {
  unsigned long long a, b;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(a), "=l"(b)
               : "l"(p));
  return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}
__device__ __forceinline__ void st_word(uint4* p, float x, float y, float z, unsigned tag) {
  const unsigned long long a = __float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
  const unsigned long long b = __float_as_uint(z) | ((unsigned long long)tag << 32);
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(a),
               "l"(b));
}

// Copies 16 bytes from global to shared memory without a register, or writes
// zeros (on = false); the copying thread may read them after copies_wait.
__device__ __forceinline__ void copy16(float* dst, const float* src, bool on) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
}
// The same for 8 bytes.
__device__ __forceinline__ void copy8(float* dst, const float* src, bool on) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(on ? 8 : 0) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The larger of a and b, NaN if either is.
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
// The stability monitor where a norm may be near 1e25: squares scaled by
// 2^-80, which neither over- nor underflow there.  NaN comes back as +inf.
__device__ __forceinline__ float norm_sq(float a, float b) {
  const float s = 8.271806e-25f;  // 2^-80
  return fmaf(a * s, a * s, (b * s) * (b * s));
}
__device__ __forceinline__ float norm_of_sq(float q) { return nan_to_inf(sqrtf(q) * 1.2089258e24f); }

// Called every few unsuccessful polls: false once the limit has passed or
// any tile has given up.  (keep_polling, inlined: a call would have the whole
// state saved around it.)
__device__ __forceinline__ bool poll_again(Ctl* ctl, unsigned long long limit_ns, unsigned long long& t0) {
  const unsigned long long now = res::res_timer_ns();
  if (t0 == 0) t0 = now;
  if (*(volatile int*)&ctl->err) return false;
  if (now - t0 > limit_ns) {
    atomicExch(&ctl->err, 1);
    return false;
  }
  return true;
}

}  // namespace
}  // namespace tile2
}  // namespace sfd

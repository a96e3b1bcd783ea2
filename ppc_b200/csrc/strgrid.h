// String-proximity table: an exact, conservative pre-test for the DOM search.
//
// The reference's DOM search (gpu/pro.cu:577-672) visits, for every propagation step, the
// strings of the skewed search cells (about 62 m wide) that the step's horizontal extent
// touches and tests each string's cylinder against the step's segment.  On the full
// detector that is about two strings per step, while fewer than 0.2% of steps pass a
// cylinder test at all.  This table lets a step prove, with one shared-memory load and a
// distance test (a cylinder test near a string), that the search would find nothing:
//
//   * lines that share an axis (a string split into several lines, axes equal up to
//     rounding) form a group, whose disc covers each line's search disc (the search radius
//     already includes the hole-ice radius);
//   * a grid of square cells covers the groups' horizontal footprint plus `margin` on every
//     side; each cell holds the group nearest to it and a lower bound on the squared distance
//     from any point of the cell to the widened disc (radius + kReachPad) of every OTHER group.
//
// A step from r, of length sca along n, reaches horizontally no farther than
// L = sca sqrt(1 - nz^2) from r.  If L is below the cell's clearance no other group can be
// reached.  The nearest group is then out of reach when r lies farther than rw + sca from
// its axis (a ball test, no square root); otherwise it is tested with the reference's
// cylinder arithmetic on the widened radius.  A string that the reference's test accepts is within its radius of the
// segment, so the widened test accepts it too: the widening changes the test's
// discriminant by 0.09 np m^2, against a rounding of at most 1e-3 np m^2 for strings
// within 120 m of the segment.  When nothing can be reached the reference's search would
// find nothing -- no DOM candidate, no hole-ice column -- so skipping it leaves the step
// bit for bit unchanged.  Otherwise (and for near-vertical or non-finite steps) the
// reference's search runs in full, in its own order.
#pragma once
#include <stdint.h>
#if !defined(__CUDA_ARCH__)
#include <cmath>
#include <cstring>
#endif

#include "ppcb_types.h"

#if defined(__CUDACC__)
#define PPCB_SG_HD __host__ __device__ __forceinline__
#else
#define PPCB_SG_HD inline
#endif

namespace ppcb {

constexpr float kReachPad = 0.05f;      // [m] added to every group's radius
constexpr int kSgMaxCells = 16384;      // cells (two bytes each): 32 KiB of shared memory
constexpr float kSgMinNp = 1e-4f;       // 1 - nz^2 below this: full search

// Table geometry (a kernel parameter).  Point (x, y) lies in column
// round(clamp(x su + ou, 0, 1) cu), row likewise: a cell's square is centred on its number.  The
// clamp puts a point outside the grid into a border cell; the clearances hold for it, since it
// is farther from every group than the border point nearest to it.  The host widens a cell's
// square by two millimetres on every side to cover the rounding of those products.
struct StrGridParams {
  float su, ou, sv, ov;        // 1 / ((cells - 1) x cell size) and -(centre of the first cell) times it
  float cu, cv;                // cells - 1, per row and column
  int32_t nx, ny, on, base;    // cells per row, rows; on = 0: no strings; -kSgMagicBits (nx + 1)
};

// Adding 1.5 x 2^23 leaves the nearest integer in a float's low bits.
constexpr float kSgMagic = 12582912.f;
constexpr int32_t kSgMagicBits = 0x4b400000;

// A cell entry: the group in the low byte; above it the upper bits of the squared clearance
// as a float (five of the exponent, from 2^-16, and three of the mantissa).  Multiplied by 4096
// the entry is that float, the group's bits in the mantissa below, which the host allows for.
constexpr uint32_t kSgClearBase = 0x37800000u;

// One group as the pre-test reads it: axis and widened radius.  After the groups the
// table holds a sentinel (an axis at 1e30 m, never within reach), the entry of a cell
// that has no nearest group.
struct StrGroup {
  float x, y, rw, pad_;
};

// The reference's cylinder test (gpu/pro.cu:601-607) on the widened radius: true when the
// segment from (rx, ry) along (nx, ny) (np = 1 - nz^2 >= kSgMinNp) of length sca may meet
// the group's cylinder.
PPCB_SG_HD bool sg_group_near(const StrGroup& G, float rx, float ry, float nx, float ny, float np, float sca) {
  const float dx = G.x - rx, dy = G.y - ry;
  const float c = dx * dx + dy * dy;
  const float b = nx * dx + ny * dy;
  const float D = b * b - (c - G.rw * G.rw) * np;
  if (!(D >= 0)) return !(D < 0);  // NaN: may reach
  const float q = sqrtf(D);
  return b + q >= -0.01f && b - q <= sca * np + 0.01f;
}

PPCB_SG_HD float sg_float(uint32_t bits) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(bits);
#else
  float f;
  std::memcpy(&f, &bits, 4);
  return f;
#endif
}

// The cell of a point, as an index into the entries.
PPCB_SG_HD int sg_cell(const StrGridParams& g, float rx, float ry) {
#if defined(__CUDA_ARCH__)
  const float u = __saturatef(fmaf(rx, g.su, g.ou)), v = __saturatef(fmaf(ry, g.sv, g.ov));  // NaN: 0
  return (int)(__float_as_uint(fmaf(v, g.cv, kSgMagic)) * (uint32_t)g.nx + __float_as_uint(fmaf(u, g.cu, kSgMagic)) +
               (uint32_t)g.base);  // unsigned: kSgMagicBits (nx + 1) wraps around, base takes it off again
#else
  const float fu = std::fma(rx, g.su, g.ou), fv = std::fma(ry, g.sv, g.ov);
  const float u = fu > 0 ? (fu < 1 ? fu : 1.f) : 0.f, v = fv > 0 ? (fv < 1 ? fv : 1.f) : 0.f;
  const int iu = (int)(std::fma(u, g.cu, kSgMagic) - kSgMagic), iv = (int)(std::fma(v, g.cv, kSgMagic) - kSgMagic);
  return iv * g.nx + iu;
#endif
}

// Whether the step may reach a string's cylinder (the full search must run).  `Tab`
// supplies cell(k) (the 16-bit cell entry) and group(m).  Host and device evaluate it with the
// same IEEE operations.  The common answer, no, comes from one straight line of instructions:
// no step but the rare one branches, and the cell index needs no conversion to integers
// (against a test with early exits and conversions: 1e3 photons 281 -> 273 us, 3e7 24930 -> 24610).
template <class Tab>
PPCB_SG_HD bool sg_may_reach(const StrGridParams& g, const Tab& t, float rx, float ry, float nx, float ny, float nz,
                             float sca) {
  if (!g.on) return false;
  const float np = 1 - nz * nz;
  const float L2 = sca * sca * np;  // squared horizontal reach of the step
  const uint32_t e = t.cell(sg_cell(g, rx, ry));
  // Near-vertical steps go to the full search: there 1 - nz^2 rounds to (nearly) zero and
  // the reference's cylinder test accepts strings at any distance (its discriminant is
  // b^2 - (c - r^2) np), which matters when hole ice is on (gpu/pro.cu:655-669).  About
  // one step in 2e4 of an isotropic photon is that steep.
  const bool other = !(np >= kSgMinNp) | !(L2 < sg_float(e * 4096u + kSgClearBase));  // another group in reach
  const StrGroup& G = t.group((int)(e & 0xff));
  const float dx = G.x - rx, dy = G.y - ry, w = G.rw + sca;
  if (!(other | !(dx * dx + dy * dy > w * w))) return false;  // the nearest axis is farther than rw + sca
  return other || sg_group_near(G, rx, ry, nx, ny, np, sca);
}

}  // namespace ppcb

// Ice-layer tilt: depth shift of the layer isochrons at (x, y, z), gpu/pro.cu:168-264.
// One implementation for the kernel and the host tools.  Every operation is an IEEE
// round-to-nearest step without contraction (explicit intrinsics on the device; the host
// code is compiled with -ffp-contract=off), so the device and the host agree bit for bit
// and the result matches an IEEE build of the reference for identical positions.
//
// `Tab` supplies interval(nr) (the 1-d map interval, tilt_interval below), span(j) (its
// ends, width and reciprocal width), rstep(i) (reciprocal 2-d grid steps), mcol(x, y) (2-d
// map column, -1 = none) and lp(i, k) (shift and slope of map i at depth point k, as float2),
// and the constants kRecip (the reciprocals may be used, tilt_quot) and kConstantLayers
// (no variable layer thickness).
#pragma once
#include <vector_types.h>

#include <cmath>
#include <cstring>

#include "ppcb_types.h"
#include "strgrid.h"

#if defined(__CUDACC__)
#define PPCB_HD __host__ __device__ __forceinline__
#else
#define PPCB_HD inline
#endif

#if defined(__CUDA_ARCH__)
#define PPCB_ADD(a, b) __fadd_rn((a), (b))
#define PPCB_SUB(a, b) __fsub_rn((a), (b))
#define PPCB_MUL(a, b) __fmul_rn((a), (b))
#define PPCB_DIV(a, b) __fdiv_rn((a), (b))
#define PPCB_FLOOR_I(x) __float2int_rd(x)
#else
#include <cmath>
#define PPCB_ADD(a, b) ((a) + (b))
#define PPCB_SUB(a, b) ((a) - (b))
#define PPCB_MUL(a, b) ((a) * (b))
#define PPCB_DIV(a, b) ((a) / (b))
#define PPCB_FLOOR_I(x) ((int)floorf(x))
#endif

namespace ppcb {

PPCB_HD int tmin(int a, int b) { return b < a ? b : a; }
PPCB_HD int tmax(int a, int b) { return a < b ? b : a; }

// The quotient a / b, correctly rounded, where y is 1 / b correctly rounded (0: not usable).
// Two quotient steps with exact fused remainders; the second starts from a quotient within
// one unit in the last place, so its result is the rounded quotient (Markstein, IBM J. Res.
// Dev. 34, 1990).  Five instructions instead of a full division, whose divisor changes
// with the map only: the same bits in 1.2e9 random quotients and in the index tests.
PPCB_HD float tilt_quot(float a, float b, float y) {
#if defined(__CUDA_ARCH__)
  const float q0 = __fmul_rn(a, y);
  const float q1 = __fmaf_rn(__fmaf_rn(-b, q0, a), y, q0);
  return __fmaf_rn(__fmaf_rn(-b, q1, a), y, q1);
#else
  (void)y;
  return PPCB_DIV(a, b);
#endif
}

// Whether 1 / b may stand for b in tilt_quot: no overflow or underflow on the way.
inline bool tilt_recip_ok(float b) { return b > 1e-6f && b < 1e6f; }

// What the kernel uses instead of divisions by the maps' steps and of a search among the 1-d
// radii; on = 0 where a map does not allow it (a single map, steps out of range, radii closer
// than a cell).  The 1-d interval of nr comes from cell round(clamp(nr scale + off, 0, 1) x
// (kTiltCells - 1)), which holds the only radius that may lie in it and the interval below.
// The cells are numbered from the outermost inwards (scale < 0): a NaN, which the clamp turns
// into 0, falls into the outermost cell, and its interval is the last one, as in the search.
constexpr int kTiltCells = 64;
struct TiltFast {
  float scale, off;
  float rstep[2];  // reciprocal 2-d grid steps
  int32_t on;
};

// 1-d map interval of nr: the first j >= 1 with nr < lr[j], or j = lnum - 1.  The radii are
// non-decreasing (checked when loaded), so that is 1 + #{k in [1, lnum-2] : !(nr < lr[k])};
// NaN counts as "not below", as in the search loop.
template <class Radii>
PPCB_HD int tilt_interval(int lnum, const Radii& lr, float nr) {
  int j = 1;
  if (lnum >= 2) {
    for (int k = 1; k < lnum - 1; k++) j += !(nr < lr(k));
  } else {
    for (; j < PPCB_LMAX; j++) if (nr < lr(j)) break;
    if (j >= PPCB_LMAX) j = PPCB_LMAX - 1;  // a single-map table would run off the end
  }
  return j;
}

// The same from the cells.
PPCB_HD int tilt_cell_interval(const TiltFast& f, const float2* cells, float nr) {
#if defined(__CUDA_ARCH__)
  const float u = __saturatef(fmaf(nr, f.scale, f.off));  // NaN: 0
  const float2 c = cells[__float_as_int(fmaf(u, kTiltCells - 1.f, kSgMagic)) - kSgMagicBits];
  return __float_as_int(c.y) + !(nr < c.x);
#else
  const float v = std::fma(nr, f.scale, f.off), u = v > 0 ? (v < 1 ? v : 1.f) : 0.f;
  const float2 c = cells[(int)(std::fma(u, kTiltCells - 1.f, kSgMagic) - kSgMagic)];
  int j;
  std::memcpy(&j, &c.y, sizeof(j));
  return j + !(nr < c.x);
#endif
}

// The cells over the inner radii lr[1..lnum-2] and a metre on either side: per cell the only
// radius that may lie in it (none: infinity, in the outermost cell minus infinity) and the
// interval below it.  A cell is widened by a hundredth of itself for the rounding of a point's
// cell number.  False where the map does not allow it.
inline bool tilt_cells(const float* lr, int lnum, TiltFast& f, float2* cells) {
  if (lnum < 2) return false;
  for (int k = 1; k < lnum; k++)
    if (!tilt_recip_ok(lr[k] - lr[k - 1])) return false;
  const double lo = lnum > 2 ? lr[1] - 1.0 : lr[0], hi = lnum > 2 ? lr[lnum - 2] + 1.0 : lr[1];
  const double w = (hi - lo) / (kTiltCells - 1);
  // a point's cell number is off by less than 63 (2 |off| + 2) / 2^24 of a cell, which has to be
  // within a hundredth
  if (std::fmax(std::fabs(lo), std::fabs(hi)) > 1000 * (hi - lo)) return false;
  f.scale = (float)(-1 / (hi - lo));
  f.off = (float)(hi / (hi - lo));
  for (int c = 0; c < kTiltCells; c++) {
    int below = 0, inside = 0;
    for (int k = 1; k < lnum - 1; k++) {
      if (c < kTiltCells - 1 && lr[k] < hi - (c + 0.51) * w) below++;
      else if (c == 0 || lr[k] <= hi - (c - 0.51) * w) inside++;
    }
    if (inside > 1) return false;
    const int j = inside || c > 0 ? 1 + below : below;
    std::memcpy(&cells[c].y, &j, sizeof(j));
    cells[c].x = inside ? lr[j] : c > 0 ? INFINITY : -INFINITY;
  }
  return true;
}

// 1-d: interpolate between the two maps bracketing the distance along 225 deg
template <class Tab>
PPCB_HD float zshift_1d_t(const ppcb_params& d, const Tab& t, float rx, float ry, float rz, float& dz) {
  {
    float nr = PPCB_SUB(PPCB_ADD(PPCB_MUL(d.lnx, rx), PPCB_MUL(d.lny, ry)), d.r0);
    const int j = t.interval(nr);
    const float4 sp = t.span(j);  // lr[j-1], lr[j], their difference, its reciprocal
    float z = PPCB_MUL(PPCB_SUB(rz, d.lmin), d.lrdz);
    int i = j - 1, k = tmin(tmax(PPCB_FLOOR_I(z), 0), d.lpts);
    const float2 pi = t.lp(i, k), pj = t.lp(j, k);
    const float ax = PPCB_SUB(nr, sp.x), ay = PPCB_SUB(sp.y, nr);
    const float wx = Tab::kRecip ? tilt_quot(ax, sp.z, sp.w) : PPCB_DIV(ax, sp.z);
    const float wy = Tab::kRecip ? tilt_quot(ay, sp.z, sp.w) : PPCB_DIV(ay, sp.z);
    float qx = PPCB_ADD(PPCB_MUL(pj.x, wx), PPCB_MUL(pi.x, wy));
    float qy = PPCB_ADD(PPCB_MUL(pj.y, wx), PPCB_MUL(pi.y, wy));
    float r = PPCB_ADD(qx, PPCB_MUL(qy, PPCB_SUB(z, (float)k)));
    if (!Tab::kConstantLayers && d.vthk != 0) dz = PPCB_DIV(dz, PPCB_SUB(1.f, PPCB_MUL(d.lrdz, qy)));
    return r;
  }
}

// 2-d: barycentric interpolation on the skewed map grid
template <class Tab>
PPCB_HD float zshift_2d_t(const ppcb_params& d, const Tab& t, float rx, float ry, float rz, float& dz) {
  {
    float qx = PPCB_ADD(PPCB_MUL(d.cb[0][0], rx), PPCB_MUL(d.cb[1][0], ry));
    float qy = PPCB_ADD(PPCB_MUL(d.cb[0][1], rx), PPCB_MUL(d.cb[1][1], ry));
    qx = PPCB_SUB(qx, d.mmin[0]);
    qy = PPCB_SUB(qy, d.mmin[1]);
    qx = Tab::kRecip ? tilt_quot(qx, d.mstp[0], t.rstep(0)) : PPCB_DIV(qx, d.mstp[0]);
    qy = Tab::kRecip ? tilt_quot(qy, d.mstp[1], t.rstep(1)) : PPCB_DIV(qy, d.mstp[1]);
    const int n0 = d.mnum[0] - 1, n1 = d.mnum[1] - 1, c0 = d.mcut[0] - 1, c1 = d.mcut[1] - 1;
    const float N0 = n0, N1 = n1, C0 = c0, C1 = c1;
    // extrapolation beyond the map edges, gpu/pro.cu:200-214: six cases, none inside the map
    if (qy < 0 || qx < 0 || qy > N1 || qx > N0 || PPCB_SUB(qy, qx) > C1 || PPCB_SUB(qx, qy) > C0) {
      float x = qx, y = qy, xy;
      if (y < 0) if (PPCB_SUB(x, y) > 0 && x <= C0) { x = PPCB_DIV(PPCB_MUL(PPCB_SUB(x, y), C0), PPCB_SUB(C0, y)); y = 0; }
      if (x < 0) if (PPCB_SUB(y, x) >= 0 && y < C1) { y = PPCB_DIV(PPCB_MUL(PPCB_SUB(y, x), C1), PPCB_SUB(C1, x)); x = 0; }
      if (y > N1) if (x >= (float)(n1 - c1) && PPCB_SUB(y, x) > (float)(n1 - n0)) {
        x = PPCB_ADD((float)(n1 - c1), PPCB_DIV(PPCB_MUL((float)(n0 - (n1 - c1)), PPCB_SUB(x, (float)(n1 - c1))),
                                                PPCB_SUB(PPCB_SUB(y, (float)(n1 - n0)), (float)(n1 - c1))));
        y = N1;
      }
      if (x > N0) if (y > (float)(n0 - c0) && PPCB_SUB(y, x) <= (float)(n1 - n0)) {
        y = PPCB_ADD((float)(n0 - c0), PPCB_DIV(PPCB_MUL((float)(n1 - (n0 - c0)), PPCB_SUB(y, (float)(n0 - c0))),
                                                PPCB_SUB(PPCB_SUB(x, (float)(n0 - n1)), (float)(n0 - c0))));
        x = N0;
      }
      if (PPCB_SUB(y, x) > C1) if (y >= C1 && x < (float)(n1 - c1)) {
        xy = PPCB_SUB(PPCB_SUB(y, x), C1);
        xy = PPCB_ADD(C1, PPCB_DIV(PPCB_MUL(PPCB_ADD(PPCB_SUB(PPCB_ADD(x, y), C1), xy), (float)(n1 - c1)),
                                   PPCB_ADD((float)(n1 - c1), xy)));
        x = PPCB_SUB(xy, C1) / 2; y = PPCB_ADD(xy, C1) / 2;
      }
      if (PPCB_SUB(x, y) > C0) if (x > C0 && y <= (float)(n0 - c0)) {
        xy = PPCB_SUB(PPCB_SUB(x, y), C0);
        xy = PPCB_ADD(C0, PPCB_DIV(PPCB_MUL(PPCB_ADD(PPCB_SUB(PPCB_ADD(x, y), C0), xy), (float)(n0 - c0)),
                                   PPCB_ADD((float)(n0 - c0), xy)));
        x = PPCB_ADD(xy, C0) / 2; y = PPCB_SUB(xy, C0) / 2;
      }
      qx = x; qy = y;
    }
    int qnx0 = tmin(tmax(PPCB_FLOOR_I(qx), 0), d.mnum[0]);
    int qny0 = tmin(tmax(PPCB_FLOOR_I(qy), 0), d.mnum[1]);
    float qrx0 = PPCB_SUB(qx, (float)qnx0), qry0 = PPCB_SUB(qy, (float)qny0);
    float qrx, qry;
    int qnx, qny;
    if (qrx0 > qry0) { qrx = qrx0; qry = qry0; qnx = qnx0 + 1; qny = qny0; }
    else { qrx = qry0; qry = qrx0; qnx = qnx0; qny = qny0 + 1; }
    int cx = t.mcol(qnx0, qny0);
    int cy = t.mcol(qnx, qny);
    int cz = t.mcol(qnx0 + 1, qny0 + 1);
    float wx = PPCB_SUB(1.f, qrx), wy = PPCB_SUB(qrx, qry), wz = qry;
    float z = PPCB_MUL(PPCB_SUB(rz, d.lmin), d.lrdz);
    int k = tmin(tmax(PPCB_FLOOR_I(z), 0), d.lpts);
    float ax = 0, ay = 0;
    if (cx >= 0) { const float2 p = t.lp(cx, k); ax = PPCB_ADD(ax, PPCB_MUL(p.x, wx)); ay = PPCB_ADD(ay, PPCB_MUL(p.y, wx)); }
    if (cy >= 0) { const float2 p = t.lp(cy, k); ax = PPCB_ADD(ax, PPCB_MUL(p.x, wy)); ay = PPCB_ADD(ay, PPCB_MUL(p.y, wy)); }
    if (cz >= 0) { const float2 p = t.lp(cz, k); ax = PPCB_ADD(ax, PPCB_MUL(p.x, wz)); ay = PPCB_ADD(ay, PPCB_MUL(p.y, wz)); }
    float r = PPCB_ADD(ax, PPCB_MUL(ay, PPCB_SUB(z, (float)k)));
    if (!Tab::kConstantLayers && d.vthk != 0) dz = PPCB_DIV(dz, PPCB_SUB(1.f, PPCB_MUL(d.lrdz, ay)));
    return r;
  }
}

template <class Tab>
PPCB_HD float zshift_t(const ppcb_params& d, const Tab& t, float rx, float ry, float rz, float& dz) {
  if (d.tmod == 1) return zshift_1d_t(d, t, rx, ry, rz, dz);
  if (d.tmod == 2) return zshift_2d_t(d, t, rx, ry, rz, dz);
  return 0;
}

}  // namespace ppcb

// Grid walk of a straight ray for the matrix-free operators.
//
// trace.cuh follows the reference's arithmetic point by point (a correctly
// rounded division per crossing, a square root per segment, a merge window),
// which is what a stored matrix needs to be bit-exact.  A product only needs
// every entry's FP32 value and its pixel, so here the walk keeps the next
// crossing parameter of each grid-line family as t0 + k/|d| (one addition and
// one multiply-add per crossing), the pixel as an integer that moves by one
// line, and the length as the difference of two parameters.  The lengths
// agree with the traced ones to a few ulps of the coordinates (about 1e-13
// at N = 512), so an entry is the stored matrix's FP32 entry except where the
// length is that close to a midpoint of two FP32 values (about one in 10^6).
//
// Bound: issue and the FP64 pipe (42 % busy, 24 instructions per cell), then
// the gathers' latency.  Measured at N = 512, 180 angles x 724 rays (61 M
// entries): forward 108 us against 646 us for the traced projector; fan
// N = 1024, 180 x 1448 (203 M entries): 335 us against 1,990 us, and the
// scatter of the back projection 660 us against 2,025 us, where the L2 takes
// the atomics.
//
// The rays of dda_slow are listed when the operator is made and traced by
// trace.cuh in a launch of their own, which is skipped when there are none:
// with that code in the walk's kernel its registers cap the resident warps
// (80 registers, or 350 bytes of spills at 64).
#pragma once

#include "trace.cuh"

namespace airt {

// Warps of a walk block: the parts a block's 32 rays are split into (at most
// kDdaParts), and warps of a pixel-driven block.  Eight parts keep the chip
// full when there are few rays; four measured better with many (108 against
// 116 us and 336 against 349 us for the two problems above).
constexpr int kDdaParts = 8, kGatherWarps = 8;
inline int dda_parts(int64_t nrays) { return nrays < 32768 ? 8 : 4; }

// x rounded to the 24 bits of an FP32 value, kept in FP64 (Veltkamp's
// splitting; |x| in the normal FP32 range or 0, not at a midpoint).  Three
// FP64 operations instead of two conversions, which run at a quarter of
// their rate.
__device__ __forceinline__ double round24(double x) {
  const double c = __dmul_rn(x, 536870913.0);
  return __dsub_rn(c, __dsub_rn(c, x));
}

// Whether trace.cuh has to follow the ray:
// * nearly, but not exactly, parallel to a grid-line family (a direction
//   component below kDdaSlope of the other): its crossings with that family
//   are ill conditioned and rounding decides the pixels of long segments;
// * along the top or right grid line, where the reference's exclusion rule
//   and its pixel index apply;
// * through a corner of the image (within kEdgeGap): rounding decides whether
//   the reference's box test keeps the corner point, and with it the corner
//   pixel's segment.
constexpr double kDdaSlope = 1e-7;
constexpr double kEdgeGap = 1e-9;

__device__ __forceinline__ bool dda_slow(int N, const Ray &q) {
  const double h = 0.5 * (double)N, fa = fabs(q.a), fb = fabs(q.b);
  const double lo = fmin(fa, fb), hi = fmax(fa, fb);
  if (!(hi < INFINITY) || hi == 0.0) return true;
  if (lo == 0.0) return fabs((fb == 0.0 ? q.y0t : q.x0t) - h) < kEdgeGap;
  if (lo < kDdaSlope * hi) return true;
  const double off = fabs(q.b * q.x0t - q.a * q.y0t), tol = kEdgeGap * hi;
  return fabs(off - h * (hi + lo)) < tol || fabs(off - h * (hi - lo)) < tol;
}

// First crossing k >= kmin of a family t(k) = t0 + k*dt with t(k) > t.
__device__ __forceinline__ double first_after(double t, double t0, double dt, double inv_dt, double kmin) {
  double k = fmax(ceil((t - t0) * inv_dt), kmin);
  while (k > kmin && fma(k - 1.0, dt, t0) > t) k -= 1.0;
  while (fma(k, dt, t0) <= t) k += 1.0;
  return k;
}

// Walks part `part` of `parts` of the ray's cells and calls emit(cell, v)
// with the FP32 entry of each (as FP64); cell is the column-major pixel index, or the
// row-major one when `swap` is set.  The parts split the ray at crossings of
// its faster family, so their cells are disjoint and their union is the whole
// walk.  UNIT: (a, b) is a unit vector (to FP64 rounding).  The caller has
// excluded dda_slow rays.
template <bool UNIT, class Emit>
__device__ __forceinline__ void dda_walk(int N, Ray q, int part, int parts, bool swap, Emit &&emit) {
  const double h = 0.5 * (double)N, dN = (double)N;
  const double fa = fabs(q.a), fb = fabs(q.b);
  // Crossing k of a family: t(k) = t0 + k*dt for k = -r..N-r from the side
  // the ray enters, where k = 0 is the line next to the ray's origin (a family
  // the ray is parallel to is never crossed).  The lines that a ray close to
  // an axis crosses lie next to its origin, so their t has few ulps of itself;
  // counted from the side, t0 is near N/slope there and twice the traced
  // crossings' error came with it (N = 512, slope 1e-6: 7e-8 against 4e-8 of
  // exact arithmetic, now 4e-8).
  double tx0 = INFINITY, dtx = 0.0, rx = 0.0, ty0 = INFINITY, dty = 0.0, ry = 0.0;
  double tin = -INFINITY, tend = INFINITY;
  if (fa != 0.0) {
    dtx = 1.0 / fa;
    rx = fmin(fmax(rint((q.a > 0.0 ? q.x0t : -q.x0t) + h), 0.0), dN);
    tx0 = ((q.a > 0.0 ? rx - h : h - rx) - q.x0t) / q.a;
    tin = fma(-rx, dtx, tx0);
    tend = fma(dN - rx, dtx, tx0);
  } else if (!(q.x0t >= -h && q.x0t < h)) {
    return;
  }
  if (fb != 0.0) {
    dty = 1.0 / fb;
    ry = fmin(fmax(rint((q.b > 0.0 ? q.y0t : -q.y0t) + h), 0.0), dN);
    ty0 = ((q.b > 0.0 ? ry - h : h - ry) - q.y0t) / q.b;
    tin = fmax(tin, fma(-ry, dty, ty0));
    tend = fmin(tend, fma(dN - ry, dty, ty0));
  } else if (!(q.y0t >= -h && q.y0t < h)) {
    return;
  }
  if (!(tin < tend)) return;
  if (parts > 1) {
    // split at crossings m_p = k0 + (k1 - k0) * p / parts of the faster family
    const bool px = fa >= fb;
    const double t0 = px ? tx0 : ty0, dt = px ? dtx : dty, f = px ? fa : fb, kmin = px ? -rx : -ry;
    const double k0 = fmax(floor((tin - t0) * f), kmin), k1 = fmin(ceil((tend - t0) * f), kmin + dN);
    const double step = (k1 - k0) / (double)parts;
    if (part + 1 < parts) tend = fmin(tend, fma(floor(fma(step, (double)(part + 1), k0)), dt, t0));
    if (part > 0) {
      const double ts = fma(floor(fma(step, (double)part, k0)), dt, t0);
      tin = fmax(tin, ts);
    }
    if (!(tin < tend)) return;
  }
  double kx = 0.0, ky = 0.0, tx = INFINITY, ty = INFINITY;
  int ix, iy;
  if (fa != 0.0) {
    kx = first_after(tin, tx0, dtx, fa, -rx);
    tx = fma(kx, dtx, tx0);
    ix = q.a > 0.0 ? (int)(kx + rx) - 1 : N - (int)(kx + rx);
  } else {
    ix = (int)floor(q.x0t + h);
  }
  if (fb != 0.0) {
    ky = first_after(tin, ty0, dty, fb, -ry);
    ty = fma(ky, dty, ty0);
    iy = q.b > 0.0 ? (int)(ky + ry) - 1 : N - (int)(ky + ry);
  } else {
    iy = (int)floor(q.y0t + h);
  }
  if (ix < 0 || ix >= N || iy < 0 || iy >= N) return;
  int cell = swap ? (N - 1 - iy) * N + ix : ix * N + (N - 1 - iy);
  const int sx = (q.a > 0.0 ? 1 : -1) * (swap ? 1 : N), sy = (q.b > 0.0 ? -1 : 1) * (swap ? N : 1);
  const double nrm = UNIT ? 1.0 : sqrt(fma(q.a, q.a, q.b * q.b));
  // pieces within 1e-10 in both coordinates are no entries (the reference's
  // duplicate-point rule)
  const double tmin = 1e-10 / fmax(fa, fb);
  double tc = tin;
  do {
    const bool takex = tx <= ty;
    const double tn = takex ? tx : ty;
    const double dt = tn - tc;
    if (dt > tmin) emit(cell, round24(UNIT ? dt : dt * nrm));
    tc = tn;
    if (takex) {
      kx += 1.0;
      tx = fma(kx, dtx, tx0);
      cell += sx;
    } else {
      ky += 1.0;
      ty = fma(ky, dty, ty0);
      cell += sy;
    }
  } while (tc < tend);
}

// Whether rays of this direction read and write better in the row-major
// copy of the image: adjacent rays of a projection that run along y are
// neighbours in x, so their lanes then share sectors.
__device__ __forceinline__ bool dda_swap(const Ray &q) { return fabs(q.b) > fabs(q.a); }

// Entries of ray r (part of parts) for the products, unless the ray is one
// of the slow list: emit(cell, swapped, v).  Returns false for those.
template <bool UNIT, class Emit>
__device__ __forceinline__ bool ray_cells(const RayGeom &g, int64_t r, int part, int parts, Emit &&emit) {
  const Ray q = ray_of(g, r);
  if (dda_slow(g.N, q)) return false;
  const bool swap = dda_swap(q);
  dda_walk<UNIT>(g.N, q, part, parts, swap, [&](int cell, double v) { emit(cell, swap, v); });
  return true;
}

// The traced entries of one of the listed rays, for part 0 or 1 of 2:
// emit(column-major pixel, FP32 entry as FP64).
template <class Emit>
__device__ __forceinline__ void slow_cells(const RayGeom &g, int64_t r, bool excl, int part, Emit &&emit) {
  const int64_t nn = (int64_t)g.N * g.N;
  trace_entries_part(g.N, ray_of(g, r), excl, part, [&](int col, double v) {
    if (col >= 0 && col < nn) emit(col, (double)(float)v);
  });
}

}  // namespace airt

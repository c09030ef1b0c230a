// Pixel-driven back projection of paralleltomo without the stored matrix.
//
// Column j of A holds, for every angle, the chords that the few rays crossing
// pixel j cut from it.  For parallel rays at uniform offsets s_k = s_0 + k*D
// that set is closed form: with the ray normal (c, s) and the pixel centre at
// u = c*x + s*y along it, the chord of ray k is the trapezoid
//   min(1/p, (w - |s_k - u|) / (p*q)),  p = max(|c|,|s|), q = min(|c|,|s|),
//   w = (p + q)/2,
// and 1 for axis-parallel rays in the pixel's half-open range (the floor rule
// of paralleltomo.m:255-263).  So a pixel gathers its sum with no atomics and
// no ray walk: per angle one projection of the centre and one or two chords.
// Bound: issue (72 % of the slots, 43 % of the FP64 pipe); 173 us at N = 512,
// 180 angles x 724 rays, update included, against 651 us for the traced
// scatter with fixed-point atomics (283 us with the walk of dda.cuh).
//
// The chord's FP32 rounding is the stored entry's as in dda.cuh; the few
// entries where the reference's box test drops a segment in a corner pixel
// (dda_slow) are corrected from a list made with the operator.
#pragma once

#include "dda.cuh"

namespace airt {

struct ParAngle {
  double c, s;     // ray normal
  double w, ip;    // half width (p + q)/2 and plateau 1/p
  double ipq;      // 1/(p*q); 0: axis-parallel rays
  double k0;       // (-w - s_0)/D: the first ray of the shadow is ceil(u/D + k0)
};

struct ParGather {
  const ParAngle *ang;  // nA
  double s0, D, iD;     // offsets s0 + k*D
  int N, nA, p;
  const struct ParFix *fix;  // nfix corrections
  int nfix;
};

// Entry (ray r, pixel j) is v more than the closed form says.
struct ParFix {
  int j, r;
  double v;
};
constexpr int kParFixMax = 64;

// Closed-form chord of a ray at distance d from the pixel centre, as an FP32
// value in FP64: 0 outside the shadow and for chords within 1e-10 in both
// coordinates (no entries by the reference's duplicate-point rule).
__device__ __forceinline__ bool par_entry(double w, double ip, double ipq, double d, double &ramp) {
  ramp = (w - fabs(d)) * ipq;
  return ramp > 1e-10 * ip;
}
__device__ __forceinline__ double par_chord(double w, double ip, double ipq, double d) {
  double ramp;
  return par_entry(w, ip, ipq, d, ramp) ? round24(ramp < ip ? ramp : ip) : 0.0;
}

// sum over the angles a0, a0 + da, ... of A(ray, pixel) * u(ray) (u null:
// all ones); pixel j is the column-major index.
template <typename TU>
__device__ __forceinline__ double par_sum(const ParGather &t, const RayGeom &g, const TU *__restrict__ u, int j,
                                          int a0, int da) {
  const int ix = j / t.N, iy = t.N - 1 - (j - ix * t.N);
  const double h = 0.5 * (double)t.N;
  const double xc = (double)ix + 0.5 - h, yc = (double)iy + 0.5 - h;
  double acc = 0.0;
  for (int a = a0; a < t.nA; a += da) {
    const double2 cs = __ldg(reinterpret_cast<const double2 *>(t.ang + a));
    const double2 wi = __ldg(reinterpret_cast<const double2 *>(t.ang + a) + 1);
    const double2 qk = __ldg(reinterpret_cast<const double2 *>(t.ang + a) + 2);
    const TU *__restrict__ ua = u ? u + (int64_t)a * t.p : nullptr;
    const double c = fma(cs.y, yc, cs.x * xc);
    // first ray above the lower edge of the pixel's shadow: ceil by adding
    // 2^52 * 1.5 in round-up mode (the integer sits in the low bits)
    double kd = __dadd_ru(fma(c, t.iD, qk.y), 6755399441055744.0);
    int k = __double2loint(kd);
    kd -= 6755399441055744.0;
    if (k < 0) {
      k = 0;
      kd = 0.0;
    }
    double d = fma(kd, t.D, t.s0) - c;
    if (qk.x > 0.0) {
      // at unit spacing two rays at most; without branches their loads and
      // chords overlap.  u is read where there is an entry, and only there:
      // it may not be finite beside it
      auto add = [&] {
        double ramp;
        const bool on = par_entry(wi.x, wi.y, qk.x, d, ramp) && k < t.p;
        const double uk = !on ? 0.0 : u ? (double)__ldg(ua + k) : 1.0;
        acc = fma(round24(ramp < wi.y ? ramp : wi.y), uk, acc);
      };
#pragma unroll
      for (int q = 0; q < 2; ++q, ++k, d += t.D) add();
      for (; d < wi.x && k < t.p; ++k, d += t.D) add();
    } else {
      // axis-parallel: the pixel holds the rays whose coordinate floors to it
      const bool vert = cs.x != 0.0;  // rays along y at x = c*offset
      for (k = max(k - 1, 0), d = fma((double)k, t.D, t.s0) - c; d < wi.x + t.D && k < t.p; ++k, d += t.D) {
        const double o = __ldg(g.offsets + k);
        const double pos = __dadd_rn(vert ? __dsub_rn(__dmul_rn(cs.x, o), __dmul_rn(cs.y, 0.0))
                                          : __dadd_rn(__dmul_rn(cs.y, o), __dmul_rn(cs.x, 0.0)), h);
        if (floor(pos) == (double)(vert ? ix : iy)) acc += u ? (double)__ldg(ua + k) : 1.0;
      }
    }
  }
  return acc;
}

// The corrections of pixel j.
template <typename TU>
__device__ __forceinline__ double par_fixes(const ParGather &t, const TU *__restrict__ u, int j) {
  double acc = 0.0;
  for (int e = 0; e < t.nfix; ++e)
    if (t.fix[e].j == j) acc = fma(t.fix[e].v, u ? (double)u[t.fix[e].r] : 1.0, acc);
  return acc;
}

}  // namespace airt

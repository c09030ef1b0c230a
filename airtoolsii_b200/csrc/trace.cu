// GPU system-matrix generation and matrix-free projectors for the
// paralleltomo / fanlineartomo / fancurvedtomo / seismictomo geometries (and
// the matrix-free products of sphericaltomo, whose matrix is in sphere.cu).
//
//  * generate_matrix: two passes over the rays (count, then fill) with an
//    exclusive scan in between give the CSR over rays; the CSC follows by a
//    stable transposition.  Row entries keep the ray order of the trace.
//    Replaces testprobs/paralleltomo.m:112-301, fanlineartomo.m:141-358 and
//    seismictomo.m:96-287 (isMatrix = 1).
//  * apply_matrix_free: forward projection (the grid walk of dda.cuh, a ray
//    in parts of 4 or 8 threads) and back projection (parallel beams: a gather
//    per pixel, gather.cuh; the others: a scatter in 64-bit fixed point, so
//    the result does not depend on the order in which rays arrive), as the
//    isMatrix = 0 handles of paralleltomo.m:280-288 do.  Entry values are
//    rounded to FP32 as the stored matrix holds them; where a length lies at a
//    rounding boundary (about one entry in a million) the two differ by one
//    FP32 unit in the last place.  sphericaltomo and rays the walk refuses are
//    traced by the tracer of trace.cuh.
#include <algorithm>
#include <climits>
#include <cstring>

#include <vector>

#include "common.cuh"
#include "gather.cuh"
#include "spmv.cuh"
#include "stream.cuh"
#include "trace.cuh"

namespace airt {

ParGather par_gather_of(const Problem &P);

namespace {

__global__ void k_trace_count(RayGeom g, int64_t nrays, bool excl, int64_t *__restrict__ counts,
                              int *__restrict__ bad) {
  const int64_t nn = (int64_t)g.N * g.N;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrays;
       r += (int64_t)gridDim.x * blockDim.x) {
    const Ray q = ray_of(g, r);
    int64_t c = 0;
    trace_entries(g.N, q, excl, [&](int col, double) {
      if (col < 0 || col >= nn) atomicExch(bad, 1);
      else ++c;
    });
    counts[r] = c;
  }
}

__global__ void k_trace_fill(RayGeom g, int64_t nrays, bool excl, const int64_t *__restrict__ rp,
                             int *__restrict__ ci, float *__restrict__ rv) {
  const int64_t nn = (int64_t)g.N * g.N;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrays;
       r += (int64_t)gridDim.x * blockDim.x) {
    const Ray q = ray_of(g, r);
    int64_t pos = rp[r];
    const int64_t end = rp[r + 1];
    trace_entries(g.N, q, excl, [&](int col, double v) {
      if (col >= 0 && col < nn && pos < end) {
        ci[pos] = col;
        rv[pos] = (float)v;
        ++pos;
      }
    });
  }
}

__global__ void k_mf_forward(RayGeom g, int64_t nrays, bool excl, const double *__restrict__ x,
                             double *__restrict__ y) {
  const int64_t nn = (int64_t)g.N * g.N;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrays;
       r += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    row_entries(g, r, excl, [&](int col, double v) {
      if (col >= 0 && col < nn) acc = fma((double)(float)v, x[col], acc);
    });
    y[r] = acc;
  }
}

// ---- back projection in fixed point
// FP64 atomics add the rays' terms in whatever order the rays arrive, so the
// last bits of a back projection would change from run to run.  Instead
// every term (float)v * u is rounded once to an integer multiple of 2^-s and
// added as a 64-bit integer, which is associative.  s is chosen per call so
// that no sum can leave +-2^62: with kbound = T * max|v| (T the power of two
// at or above the most terms any pixel receives, max|v| a bound on the
// entries) and 2^e > kbound * max|u|, each term is below 2^62 / T in
// magnitude when scaled by 2^(62-e).  The quantum is then 2^-52 of the
// largest possible term for T = 2^10 -- FP64 accuracy -- and the result is
// bitwise the same on every run.
// 2^e > kbound * umax; INT_MIN when the product is 0 (the sums are 0),
// INT_MAX when it is not finite (the sums are NaN).
__device__ __forceinline__ int fx_exponent(double kbound, double umax) {
  const double prod = kbound * umax;
  if (!(prod < INFINITY)) return INT_MAX;
  return prod > 0.0 ? ilogb(prod) + 1 : INT_MIN;
}

__global__ void k_absmax(int64_t n, const double *__restrict__ u, const float *__restrict__ u32,
                         unsigned long long *__restrict__ bits, const int *stop_flag) {
  if (stop_flag && *(volatile const int *)stop_flag) return;
  double m = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    m = fmax(m, fabs(u ? u[i] : (double)u32[i]));
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.0)  // nonnegative doubles order as their bits
    atomicMax(bits, (unsigned long long)__double_as_longlong(m));
}

// The terms of sphericaltomo's circles (one thread per circle).
template <typename TU>
__global__ void k_mf_adjoint_fx(RayGeom g, int64_t nrays, bool excl, const TU *__restrict__ u,
                                long long *__restrict__ acc, double kbound,
                                const unsigned long long *__restrict__ umax_bits,
                                const int *stop_flag) {
  if (stop_flag && *(volatile const int *)stop_flag) return;
  const int e = fx_exponent(kbound, __longlong_as_double((long long)*umax_bits));
  if (e == INT_MIN || e == INT_MAX) return;  // u == 0 (result 0) or not finite (NaN)
  const double sc = ldexp(1.0, 62 - e);
  const int64_t nn = (int64_t)g.N * g.N;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrays;
       r += (int64_t)gridDim.x * blockDim.x) {
    const double ur = (double)u[r];
    if (ur == 0.0) continue;
    row_entries(g, r, excl, [&](int col, double v) {
      if (col >= 0 && col < nn) {
        const long long t = __double2ll_rn(__dmul_rn((double)(float)v, ur) * sc);
        atomicAdd(reinterpret_cast<unsigned long long *>(acc + col), (unsigned long long)t);
      }
    });
  }
}

// The terms of straight rays: warp w of a block walks part w of the block's
// 32 rays (dda.cuh), so that the lanes of a warp scatter to neighbouring
// pixels; walks along y go to the row-major sums acct.  u null: all ones.
template <bool UNIT, typename TU>
__global__ void __launch_bounds__(32 * kDdaParts, 4) k_dda_adjoint_fx(RayGeom g, int nrays, const TU *__restrict__ u,
                                 unsigned long long *__restrict__ acc,
                                 unsigned long long *__restrict__ acct, double kbound,
                                 const unsigned long long *__restrict__ umax_bits, const int *stop_flag) {
  if (stop_flag && *(volatile const int *)stop_flag) return;
  const int e = fx_exponent(kbound, umax_bits ? __longlong_as_double((long long)*umax_bits) : 1.0);
  if (e == INT_MIN || e == INT_MAX) return;  // u == 0 (result 0) or not finite (NaN)
  const int r = blockIdx.x * 32 + (threadIdx.x & 31);
  if (r >= nrays) return;
  const double us = (u ? (double)u[r] : 1.0) * ldexp(1.0, 62 - e);  // exact scaling
  if (us == 0.0) return;
  ray_cells<UNIT>(g, r, threadIdx.x >> 5, blockDim.x >> 5, [&](int cell, bool swapped, double v) {
    const long long t = __double2ll_rn(__dmul_rn(v, us));
    atomicAdd((swapped ? acct : acc) + cell, (unsigned long long)t);
  });
}

// The terms of the listed slow rays, two threads per ray.
template <typename TU>
__global__ void __launch_bounds__(64)
    k_slow_adjoint_fx(RayGeom g, int nslow, bool excl, const int *__restrict__ rays, const TU *__restrict__ u,
                      unsigned long long *__restrict__ acc, double kbound,
                      const unsigned long long *__restrict__ umax_bits, const int *stop_flag) {
  if (stop_flag && *(volatile const int *)stop_flag) return;
  const int e = fx_exponent(kbound, umax_bits ? __longlong_as_double((long long)*umax_bits) : 1.0);
  if (e == INT_MIN || e == INT_MAX) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >> 1 >= nslow) return;
  const int r = rays[t >> 1];
  const double us = (u ? (double)u[r] : 1.0) * ldexp(1.0, 62 - e);
  if (us == 0.0) return;
  slow_cells(g, r, excl, t & 1, [&](int cell, double v) {
    atomicAdd(acc + cell, (unsigned long long)__double2ll_rn(__dmul_rn(v, us)));
  });
}

// out = acc + transpose(acct) as integers, then FP64 (out and acc are the
// same array).
__global__ void k_fx_merge_f64(int N, double *__restrict__ out, const long long *__restrict__ acct,
                               double kbound, const unsigned long long *__restrict__ umax_bits,
                               const int *stop_flag) {
  if (stop_flag && *(volatile const int *)stop_flag) return;
  __shared__ long long t[32][33];
  const int e = fx_exponent(kbound, umax_bits ? __longlong_as_double((long long)*umax_bits) : 1.0);
  const double inv = e == INT_MIN ? 0.0 : e == INT_MAX ? __longlong_as_double(0x7ff8000000000000LL)
                                                       : ldexp(1.0, e - 62);
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;  // columns (x) and rows of the tile
  for (int q = threadIdx.y; q < 32; q += blockDim.y)
    if (r0 + q < N && c0 + threadIdx.x < N) t[q][threadIdx.x] = acct[(int64_t)(r0 + q) * N + c0 + threadIdx.x];
  __syncthreads();
  long long *acc = reinterpret_cast<long long *>(out);
  for (int q = threadIdx.y; q < 32; q += blockDim.y)
    if (c0 + q < N && r0 + threadIdx.x < N) {
      const int64_t j = (int64_t)(c0 + q) * N + r0 + threadIdx.x;
      out[j] = (double)(acc[j] + t[threadIdx.x][q]) * inv;
    }
}

// dst = transpose(src), N x N.
template <typename T>
__global__ void k_transpose_img(int N, const T *__restrict__ src, T *__restrict__ dst) {
  __shared__ T t[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int q = threadIdx.y; q < 32; q += blockDim.y)
    if (c0 + q < N && r0 + threadIdx.x < N) t[q][threadIdx.x] = src[(int64_t)(c0 + q) * N + r0 + threadIdx.x];
  __syncthreads();
  for (int q = threadIdx.y; q < 32; q += blockDim.y)
    if (r0 + q < N && c0 + threadIdx.x < N) dst[(int64_t)(r0 + q) * N + c0 + threadIdx.x] = t[threadIdx.x][q];
}

// y = A*x over straight rays: the parts of a ray are added in order.
template <bool UNIT>
__global__ void k_dda_forward(RayGeom g, int nrays, const double *__restrict__ x,
                              const double *__restrict__ xt, double *__restrict__ y) {
  __shared__ double sh[kDdaParts][32];
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5, parts = blockDim.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  double acc = 0.0;
  bool walked = false;
  if (r < nrays)
    walked = ray_cells<UNIT>(g, r, part, parts, [&](int cell, bool swapped, double v) {
      acc = fma(v, __ldg((swapped ? xt : x) + cell), acc);
    });
  sh[part][lane] = acc;
  __syncthreads();
  if (part == 0 && walked) {
    for (int q = 1; q < parts; ++q) acc += sh[q][lane];
    y[r] = acc;
  }
}

// The listed slow rays' rows of y = A*x (x given) or of s2 and s1 (two
// threads per ray).
__global__ void __launch_bounds__(64)
    k_slow_rows(RayGeom g, int nslow, bool excl, const int *__restrict__ rays, const double *__restrict__ x,
                double *__restrict__ y, double *__restrict__ s2, double *__restrict__ s1) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, e = t >> 1;
  double a = 0.0, a2 = 0.0, a1 = 0.0;
  if (e < nslow)
    slow_cells(g, rays[e], excl, t & 1, [&](int cell, double v) {
      if (x) a = fma(v, x[cell], a);
      a2 = fma(v, v, a2);
      a1 += v;
    });
  a += __shfl_xor_sync(0xffffffffu, a, 1);
  a2 += __shfl_xor_sync(0xffffffffu, a2, 1);
  a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
  if (e >= nslow || (t & 1)) return;
  if (y) y[rays[e]] = a;
  if (s2) s2[rays[e]] = a2;
  if (s1) s1[rays[e]] = a1;
}

// Lists the slow rays and counts them in *cnt (at most m).
__global__ void k_list_slow(RayGeom g, int nrays, int *__restrict__ list, int *__restrict__ cnt) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < nrays && dda_slow(g.N, ray_of(g, r))) list[atomicAdd(cnt, 1)] = r;
}

// Row sums of v^2 and |v| over straight rays.
template <bool UNIT>
__global__ void k_dda_row_stats(RayGeom g, int nrays, double *__restrict__ s2,
                                double *__restrict__ s1) {
  __shared__ double sh2[kDdaParts][32], sh1[kDdaParts][32];
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5, parts = blockDim.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  double a2 = 0.0, a1 = 0.0;
  bool walked = false;
  if (r < nrays)
    walked = ray_cells<UNIT>(g, r, part, parts, [&](int, bool, double v) {
      a2 = fma(v, v, a2);
      a1 += v;
    });
  sh2[part][lane] = a2;
  sh1[part][lane] = a1;
  __syncthreads();
  if (part == 0 && walked) {
    for (int q = 1; q < parts; ++q) {
      a2 += sh2[q][lane];
      a1 += sh1[q][lane];
    }
    if (s2) s2[r] = a2;
    if (s1) s1[r] = a1;
  }
}

// Pixel-driven back projection: warp w of a block sums the angles w, w +
// warps, ... of the block's 32 pixels; the warps' sums are added in order.
template <typename TU>
__global__ void __launch_bounds__(32 * kGatherWarps, 5)
    k_par_gather(ParGather t, RayGeom g, int n, const TU *__restrict__ u, double *__restrict__ out,
                 const int *stop_flag) {
  if (stop_flag && *(volatile const int *)stop_flag) return;
  __shared__ double sh[kGatherWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  double acc = j < n ? par_sum(t, g, u, j, w, kGatherWarps) : 0.0;
  sh[w][lane] = acc;
  __syncthreads();
  if (w == 0 && j < n) {
    for (int q = 1; q < kGatherWarps; ++q) acc += sh[q][lane];
    out[j] = acc + par_fixes(t, u, j);
  }
}

// The corrections of the rays through the image's corners: for each listed
// ray and each of its pixels, the traced entry less the closed form's (which
// gives a pixel the reference dropped, too).  cand: the corner pixels.
__global__ void k_par_fixes(ParGather t, RayGeom g, int nslow, const int *__restrict__ rays,
                            ParFix *__restrict__ fix, int *__restrict__ cnt) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= 4 * nslow) return;
  const int r = rays[q >> 2], c = q & 3, N = t.N;
  const int ix = c & 1 ? N - 1 : 0, iy = c & 2 ? N - 1 : 0;
  if (N == 1 && c) return;
  const int j = ix * N + (N - 1 - iy), a = r / t.p, k = r - a * t.p;
  const ParAngle A = t.ang[a];
  if (!(A.ipq > 0.0)) return;
  double v = 0.0;
  trace_entries(N, ray_of(g, r), true, [&](int col, double len) {
    if (col == j) v += (double)(float)len;
  });
  const double h = 0.5 * (double)N;
  const double d = fma((double)k, t.D, t.s0) - fma(A.s, (double)iy + 0.5 - h, A.c * ((double)ix + 0.5 - h));
  const double f = par_chord(A.w, A.ip, A.ipq, d);
  if (v == f) return;
  const int e = atomicAdd(cnt, 1);
  if (e < kParFixMax) fix[e] = ParFix{j, r, v - f};
}

// Fixed-point sums back to FP64, in place (acc and out are the same array).
__global__ void k_fx_to_f64(int64_t n, double *__restrict__ out, double kbound,
                            const unsigned long long *__restrict__ umax_bits, const int *stop_flag) {
  if (stop_flag && *(volatile const int *)stop_flag) return;
  const int e = fx_exponent(kbound, umax_bits ? __longlong_as_double((long long)*umax_bits) : 1.0);
  const double inv = e == INT_MIN ? 0.0 : e == INT_MAX ? __longlong_as_double(0x7ff8000000000000LL)
                                                       : ldexp(1.0, e - 62);
  long long *acc = reinterpret_cast<long long *>(out);
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * blockDim.x)
    out[j] = (double)acc[j] * inv;
}

// Terms each pixel receives and the largest entry, over every ray (the
// bounds of the fixed-point scale); counts as the sums are scattered.
__global__ void k_mf_emit_stats(RayGeom g, int64_t nrays, bool excl, int *__restrict__ cnt,
                                unsigned long long *__restrict__ vmax_bits) {
  const int64_t nn = (int64_t)g.N * g.N;
  double vm = 0.0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrays;
       r += (int64_t)gridDim.x * blockDim.x)
    row_entries(g, r, excl, [&](int col, double v) {
      if (col >= 0 && col < nn) {
        atomicAdd(cnt + col, 1);
        vm = fmax(vm, fabs((double)(float)v));
      }
    });
  if (vm > 0.0) atomicMax(vmax_bits, (unsigned long long)__double_as_longlong(vm));
}

__global__ void __launch_bounds__(64)
    k_slow_emit_stats(RayGeom g, int nslow, bool excl, const int *__restrict__ rays, int *__restrict__ cnt,
                      unsigned long long *__restrict__ vmax_bits) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >> 1 >= nslow) return;
  double vm = 0.0;
  slow_cells(g, rays[t >> 1], excl, t & 1, [&](int cell, double v) {
    atomicAdd(cnt + cell, 1);
    vm = fmax(vm, v);
  });
  if (vm > 0.0) atomicMax(vmax_bits, (unsigned long long)__double_as_longlong(vm));
}

template <bool UNIT>
__global__ void k_dda_emit_stats(RayGeom g, int nrays, int *__restrict__ cnt,
                                 int *__restrict__ cntt, unsigned long long *__restrict__ vmax_bits) {
  const int r = blockIdx.x * 32 + (threadIdx.x & 31);
  double vm = 0.0;
  if (r < nrays)
    ray_cells<UNIT>(g, r, threadIdx.x >> 5, blockDim.x >> 5, [&](int cell, bool swapped, double v) {
      atomicAdd((swapped ? cntt : cnt) + cell, 1);
      vm = fmax(vm, v);
    });
  for (int o = 16; o > 0; o >>= 1) vm = fmax(vm, __shfl_xor_sync(0xffffffffu, vm, o));
  if ((threadIdx.x & 31) == 0 && vm > 0.0)
    atomicMax(vmax_bits, (unsigned long long)__double_as_longlong(vm));
}

__global__ void k_max_int(int64_t n, const int *__restrict__ a, int *__restrict__ out) {
  int m = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, a[i]);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Per-ray sums (squares, absolute values, squares weighted by colw) and
// per-pixel counts and absolute sums, in one pass over the rays.
// cs1 (column sums of |v|) is accumulated in fixed point (see above) with
// max|u| = 1 and converted by k_fx_to_f64.
__global__ void k_mf_stats(RayGeom g, int64_t nrays, bool excl, double *__restrict__ s2,
                           double *__restrict__ s1, double *__restrict__ ccnt,
                           double *__restrict__ cs1, const double *__restrict__ colw,
                           double *__restrict__ s2w, double kbound) {
  const int64_t nn = (int64_t)g.N * g.N;
  const double sc = ldexp(1.0, 62 - fx_exponent(kbound, 1.0));
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrays;
       r += (int64_t)gridDim.x * blockDim.x) {
    const Ray q = ray_of(g, r);
    double a2 = 0, a1 = 0, aw = 0;
    trace_entries(g.N, q, excl, [&](int col, double v64) {
      if (col < 0 || col >= nn) return;
      const double v = (double)(float)v64;
      a2 += v * v;
      a1 += fabs(v);
      if (colw) aw += v * v * colw[col];
      if (ccnt) atomicAdd(ccnt + col, 1.0);
      if (cs1)
        atomicAdd(reinterpret_cast<unsigned long long *>(cs1) + col,
                  (unsigned long long)__double2ll_rn(fabs(v) * sc));
    });
    if (s2) s2[r] = a2;
    if (s1) s1[r] = a1;
    if (s2w) s2w[r] = aw;
  }
}

inline bool excl_of(const Problem &P) { return P.geo_kind == GEO_PARALLEL; }
inline unsigned slow_grid(const Problem &P) { return (unsigned)((2 * (int64_t)P.nslow + 63) / 64); }
inline bool straight(const Problem &P) { return P.geo_kind != GEO_SPHERE; }

// Launches KERNEL<UNIT> over the rays, dda_parts(m) warps of 32 rays per block.
#define AIRT_DDA_LAUNCH(KERNEL, ...)                                                           \
  do {                                                                                        \
    const unsigned g_ = (unsigned)((P.m + 31) / 32), t_ = 32u * dda_parts(P.m);                 \
    if (P.geo_kind == GEO_SEISMIC) KERNEL<false><<<g_, t_, 0, s>>>(P.geom(), (int)P.m, __VA_ARGS__); \
    else KERNEL<true><<<g_, t_, 0, s>>>(P.geom(), (int)P.m, __VA_ARGS__);                        \
  } while (0)

template <typename TU>
void dda_adjoint(Problem &P, const TU *u, double *out, const unsigned long long *umax, const int *stop) {
  cudaStream_t s = P.stream;
  const unsigned g_ = (unsigned)((P.m + 31) / 32), t_ = 32u * dda_parts(P.m);
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(out);
  unsigned long long *acct = reinterpret_cast<unsigned long long *>(P.fxt.p);
  AIRT_CHECK_CUDA(cudaMemsetAsync(acc, 0, P.n * sizeof(double), s));
  AIRT_CHECK_CUDA(cudaMemsetAsync(acct, 0, P.n * sizeof(double), s));
  if (P.m) {
    if (P.geo_kind == GEO_SEISMIC)
      k_dda_adjoint_fx<false, TU><<<g_, t_, 0, s>>>(P.geom(), (int)P.m, u, acc, acct, P.mf_kbound, umax, stop);
    else
      k_dda_adjoint_fx<true, TU><<<g_, t_, 0, s>>>(P.geom(), (int)P.m, u, acc, acct, P.mf_kbound, umax, stop);
    if (P.nslow)
      k_slow_adjoint_fx<TU><<<slow_grid(P), 64, 0, s>>>(P.geom(), P.nslow, excl_of(P), P.slow_rays.p, u, acc,
                                                        P.mf_kbound, umax, stop);
  }
  const unsigned tn = (unsigned)((P.N + 31) / 32);
  k_fx_merge_f64<<<dim3(tn, tn), dim3(32, 8), 0, s>>>(P.N, out, P.fxt.p, P.mf_kbound, umax, stop);
  AIRT_LAUNCH_CHECK();
}

template <typename TU>
void par_backproject(Problem &P, const TU *u, double *out, const int *stop) {
  k_par_gather<TU><<<(unsigned)((P.n + 31) / 32), 32 * kGatherWarps, 0, P.stream>>>(
      par_gather_of(P), P.geom(), (int)P.n, u, out, stop);
  AIRT_LAUNCH_CHECK();
}

// The angle records of the pixel-driven back projection, when the geometry
// takes it: parallel rays at uniform offsets (to a few ulps), every angle
// axis-parallel or inclined by at least kDdaSlope.
void par_prepare(Problem &P) {
  P.par_ok = false;
  if (P.geo_kind != GEO_PARALLEL || P.p < 2 || P.nA < 1 || P.n >= INT_MAX - 32) return;
  cudaStream_t s = P.stream;
  std::vector<double> off(P.p), c(P.nA), sn(P.nA);
  AIRT_CHECK_CUDA(cudaMemcpyAsync(off.data(), P.offsets.p, P.p * sizeof(double), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaMemcpyAsync(c.data(), P.cos_t.p, P.nA * sizeof(double), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaMemcpyAsync(sn.data(), P.sin_t.p, P.nA * sizeof(double), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  const double D = (off[P.p - 1] - off[0]) / (P.p - 1);
  // far finer rays than pixels would make a pixel's inner loop long
  if (!(D > 1.0 / 64) || !std::isfinite(D)) return;
  // ray numbers are taken in 32 bits
  if (!(std::fabs(off[0]) / D < 1e9)) return;
  // a few ulps of the offsets, but no more than shifts a chord by 1e-9 (a
  // detector of 10^6 pixels or wider: its inner rays are finer than its ends)
  const double tol =
      std::fmin(8 * 2.2e-16 * std::fmax(std::fabs(off[0]), std::fabs(off[P.p - 1])), 1e-9);
  for (int k = 0; k < P.p; ++k)
    if (!(std::fabs(off[k] - (off[0] + k * D)) <= tol)) return;
  std::vector<ParAngle> t(P.nA);
  for (int i = 0; i < P.nA; ++i) {
    const double fc = std::fabs(c[i]), fs = std::fabs(sn[i]);
    const double p = std::fmax(fc, fs), q = std::fmin(fc, fs);
    if (!(std::fabs(p * p + q * q - 1.0) < 1e-14) || (q != 0.0 && q < kDdaSlope)) return;
    t[i] = ParAngle{c[i], sn[i], 0.5 * (p + q), 1.0 / p, q != 0.0 ? 1.0 / (p * q) : 0.0,
                    (-0.5 * (p + q) - off[0]) / D};
  }
  static_assert(sizeof(ParAngle) == 6 * sizeof(double), "angle record");
  P.par_ang.upload(reinterpret_cast<const double *>(t.data()), t.size() * 6, s);
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  P.par_s0 = off[0];
  P.par_D = D;
  P.par_nfix = 0;
  if (P.nslow) {  // rays through the corners; a longer list leaves the scatter in place
    DevBuf<int> cnt;
    cnt.ensure(1);
    static_assert(sizeof(ParFix) == 2 * sizeof(double), "correction record");
    P.par_fix.ensure(2 * kParFixMax);
    AIRT_CHECK_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int), s));
    k_par_fixes<<<(unsigned)((4 * (int64_t)P.nslow + 63) / 64), 64, 0, s>>>(
        par_gather_of(P), P.geom(), P.nslow, P.slow_rays.p, reinterpret_cast<ParFix *>(P.par_fix.p), cnt.p);
    AIRT_LAUNCH_CHECK();
    int h = 0;
    AIRT_CHECK_CUDA(cudaMemcpyAsync(&h, cnt.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
    if (h > kParFixMax) return;
    // in the order of pixels and rays: the sums of two operators of one
    // geometry are the same
    std::vector<ParFix> f(h);
    if (h) {
      AIRT_CHECK_CUDA(cudaMemcpyAsync(f.data(), P.par_fix.p, h * sizeof(ParFix), cudaMemcpyDeviceToHost, s));
      AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
      std::sort(f.begin(), f.end(), [](const ParFix &x, const ParFix &y) { return x.j != y.j ? x.j < y.j : x.r < y.r; });
      P.par_fix.upload(reinterpret_cast<const double *>(f.data()), 2 * (size_t)h, s);
      AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
    }
    P.par_nfix = h;
  }
  P.par_ok = true;
}

}  // namespace

void generate_matrix(Problem &P) {
  if (P.geo_kind == GEO_SPHERE) {
    generate_sphere_matrix(P);
    return;
  }
  cudaStream_t s = P.stream;
  const RayGeom g = P.geom();
  const int64_t nrays = P.m;
  DevBuf<int64_t> counts;
  DevBuf<int> bad;
  counts.ensure(nrays);
  bad.ensure(1);
  AIRT_CHECK_CUDA(cudaMemsetAsync(bad.p, 0, sizeof(int), s));
  const unsigned grid = grid_for(nrays, 128, 16);
  k_trace_count<<<grid, 128, 0, s>>>(g, nrays, excl_of(P), counts.p, bad.p);
  AIRT_LAUNCH_CHECK();
  P.rp.ensure(nrays + 1 + kPtrPad);
  AIRT_CHECK_CUDA(cudaMemsetAsync(P.rp.p + nrays + 1, 0, kPtrPad * sizeof(int64_t), s));
  exclusive_scan_i64(counts.p, P.rp.p, nrays, s);
  int hbad = 0;
  AIRT_CHECK_CUDA(cudaMemcpyAsync(&P.nnz, P.rp.p + nrays, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaMemcpyAsync(&hbad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  AIRT_REQUIRE(!hbad, "ray trace produced a pixel index outside the image");
  P.ci.ensure(P.nnz + kPad);
  P.rv.ensure(P.nnz + kPad);
  AIRT_CHECK_CUDA(cudaMemsetAsync(P.ci.p + P.nnz, 0, kPad * sizeof(int), s));
  AIRT_CHECK_CUDA(cudaMemsetAsync(P.rv.p + P.nnz, 0, kPad * sizeof(float), s));
  k_trace_fill<<<grid, 128, 0, s>>>(g, nrays, excl_of(P), P.rp.p, P.ci.p, P.rv.p);
  AIRT_LAUNCH_CHECK();
  build_csc_from_csr(P);
  finalize_matrix(P);
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
}

void mf_prepare(Problem &P) {
  cudaStream_t s = P.stream;
  DevBuf<int> cnt, cmax;
  DevBuf<unsigned long long> vbits;
  cnt.ensure(P.n > 0 ? P.n : 1);
  cmax.ensure(1);
  vbits.ensure(1);
  AIRT_CHECK_CUDA(cudaMemsetAsync(cnt.p, 0, (P.n > 0 ? P.n : 1) * sizeof(int), s));
  AIRT_CHECK_CUDA(cudaMemsetAsync(cmax.p, 0, sizeof(int), s));
  AIRT_CHECK_CUDA(cudaMemsetAsync(vbits.p, 0, sizeof(unsigned long long), s));
  DevBuf<int> cntt, cmaxt;  // walks along y count in the row-major image
  cmaxt.ensure(1);
  AIRT_CHECK_CUDA(cudaMemsetAsync(cmaxt.p, 0, sizeof(int), s));
  if (P.m > 0 && straight(P)) {
    cntt.ensure(P.n);
    AIRT_CHECK_CUDA(cudaMemsetAsync(cntt.p, 0, P.n * sizeof(int), s));
    P.slow_rays.ensure(P.m);
    DevBuf<int> ns;
    ns.ensure(1);
    AIRT_CHECK_CUDA(cudaMemsetAsync(ns.p, 0, sizeof(int), s));
    k_list_slow<<<(unsigned)((P.m + 255) / 256), 256, 0, s>>>(P.geom(), (int)P.m, P.slow_rays.p, ns.p);
    AIRT_CHECK_CUDA(cudaMemcpyAsync(&P.nslow, ns.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
    AIRT_DDA_LAUNCH(k_dda_emit_stats, cnt.p, cntt.p, vbits.p);
    if (P.nslow)
      k_slow_emit_stats<<<slow_grid(P), 64, 0, s>>>(P.geom(), P.nslow, excl_of(P), P.slow_rays.p, cnt.p, vbits.p);
    k_max_int<<<grid_for(P.n, 256), 256, 0, s>>>(P.n, cntt.p, cmaxt.p);
  } else if (P.m > 0) {
    k_mf_emit_stats<<<grid_for(P.m, 128, 16), 128, 0, s>>>(P.geom(), P.m, excl_of(P), cnt.p,
                                                            vbits.p);
  }
  if (P.n > 0) k_max_int<<<grid_for(P.n, 256), 256, 0, s>>>(P.n, cnt.p, cmax.p);
  AIRT_LAUNCH_CHECK();
  int hmax = 0, hmaxt = 0;
  AIRT_CHECK_CUDA(cudaMemcpyAsync(&hmaxt, cmaxt.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  unsigned long long hv = 0;
  AIRT_CHECK_CUDA(cudaMemcpyAsync(&hmax, cmax.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaMemcpyAsync(&hv, vbits.p, sizeof(hv), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  double T = 1.0;  // a bound on a pixel's terms from both walks
  while (T < (double)hmax + (double)hmaxt) T *= 2.0;
  double vmax = 0.0;
  std::memcpy(&vmax, &hv, sizeof(vmax));
  P.mf_kbound = T * (vmax > 0.0 ? vmax : 1.0);
  P.mf_umax.ensure(1);
  par_prepare(P);
  // what the products and the iterations of a solve write beside their
  // operands: none of them allocates, so that they can be captured
  if (straight(P)) {
    P.x64t.ensure(P.n);
    if (!P.par_ok) P.fxt.ensure(P.n);
    if (P.nslow) P.slow_y.ensure(P.m);
  }
}

ParGather par_gather_of(const Problem &P) {
  return ParGather{reinterpret_cast<const ParAngle *>(P.par_ang.p), P.par_s0, P.par_D, 1.0 / P.par_D, P.N, P.nA,
                   P.p, reinterpret_cast<const ParFix *>(P.par_fix.p), P.par_nfix};
}

void apply_matrix_free(Problem &P, const double *d_in, double *d_out, int transp) {
  cudaStream_t s = P.stream;
  const RayGeom g = P.geom();
  if (!transp) {
    if (P.m == 0) return;
    if (straight(P)) {
      const unsigned tn = (unsigned)((P.N + 31) / 32);
      k_transpose_img<double><<<dim3(tn, tn), dim3(32, 8), 0, s>>>(P.N, d_in, P.x64t.p);
      AIRT_DDA_LAUNCH(k_dda_forward, d_in, P.x64t.p, d_out);
      if (P.nslow)
        k_slow_rows<<<slow_grid(P), 64, 0, s>>>(g, P.nslow, excl_of(P), P.slow_rays.p, d_in, d_out, nullptr,
                                                nullptr);
    } else {
      k_mf_forward<<<grid_for(P.m, 128, 16), 128, 0, s>>>(g, P.m, excl_of(P), d_in, d_out);
    }
  } else if (P.par_ok) {
    par_backproject<double>(P, d_in, d_out, nullptr);
  } else {
    AIRT_CHECK_CUDA(cudaMemsetAsync(P.mf_umax.p, 0, sizeof(unsigned long long), s));
    k_absmax<<<grid_for(P.m, 256), 256, 0, s>>>(P.m, d_in, nullptr, P.mf_umax.p, nullptr);
    if (straight(P)) {
      dda_adjoint<double>(P, d_in, d_out, P.mf_umax.p, nullptr);
    } else {
      AIRT_CHECK_CUDA(cudaMemsetAsync(d_out, 0, P.n * sizeof(double), s));
      k_mf_adjoint_fx<double><<<grid_for(P.m, 128, 16), 128, 0, s>>>(
          g, P.m, excl_of(P), d_in, reinterpret_cast<long long *>(d_out), P.mf_kbound, P.mf_umax.p, nullptr);
      k_fx_to_f64<<<grid_for(P.n, 256), 256, 0, s>>>(P.n, d_out, P.mf_kbound, P.mf_umax.p, nullptr);
    }
  }
  AIRT_LAUNCH_CHECK();
}

void row_col_stats_mf(Problem &P, double *s2, double *s1, double *colcnt, double *cols1,
                      const double *colw, double *s2w) {
  if (P.geo_kind == GEO_SPHERE) {  // a circle's hits need merging into (pixel, count) first
    sphere_stats(P, s2, s1, colcnt, cols1, colw, s2w);
    return;
  }
  cudaStream_t s = P.stream;
  // The counts of nonzeros need the traced entries (slivers count); sums do
  // not.
  if (!colcnt && !s2w) {
    if ((s2 || s1) && P.m) {
      AIRT_DDA_LAUNCH(k_dda_row_stats, s2, s1);
      if (P.nslow)
        k_slow_rows<<<slow_grid(P), 64, 0, s>>>(P.geom(), P.nslow, excl_of(P), P.slow_rays.p, nullptr, nullptr,
                                                s2, s1);
    }
    if (cols1 && P.par_ok) par_backproject<double>(P, nullptr, cols1, nullptr);
    else if (cols1) dda_adjoint<double>(P, nullptr, cols1, nullptr, nullptr);
    AIRT_LAUNCH_CHECK();
    return;
  }
  if (colcnt) AIRT_CHECK_CUDA(cudaMemsetAsync(colcnt, 0, P.n * sizeof(double), s));
  if (cols1) AIRT_CHECK_CUDA(cudaMemsetAsync(cols1, 0, P.n * sizeof(double), s));
  k_mf_stats<<<grid_for(P.m, 128, 16), 128, 0, s>>>(P.geom(), P.m, excl_of(P), s2, s1, colcnt,
                                                      cols1, colw, s2w, P.mf_kbound);
  if (cols1)
    k_fx_to_f64<<<grid_for(P.n, 256), 256, 0, s>>>(P.n, cols1, P.mf_kbound, nullptr, nullptr);
  AIRT_LAUNCH_CHECK();
}

// ---- check of the split trace: per ray, the entries of trace_entries and
// the union of trace_entries_part(0) and (1) compared by count and an
// order-independent hash of (pixel, FP64 value bits).
namespace {
__device__ __forceinline__ unsigned long long entry_hash(int col, double v) {
  unsigned long long z = (unsigned long long)__double_as_longlong(v) ^ ((unsigned long long)(unsigned)col << 1);
  z ^= z >> 33;
  z *= 0xff51afd7ed558ccdull;
  z ^= z >> 33;
  z *= 0xc4ceb9fe1a85ec53ull;
  z ^= z >> 33;
  return z;
}

__global__ void k_test_split(RayGeom g, int64_t nrays, bool excl, unsigned long long *__restrict__ bad,
                             unsigned long long *__restrict__ nsplit) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrays;
       r += (int64_t)gridDim.x * blockDim.x) {
    const Ray q = ray_of(g, r);
    unsigned long long h0 = 0, h1 = 0;
    long long c0 = 0, c1 = 0, c2 = 0;
    trace_entries(g.N, q, excl, [&](int col, double v) { h0 += entry_hash(col, v); ++c0; });
    trace_entries_part(g.N, q, excl, 0, [&](int col, double v) { h1 += entry_hash(col, v); ++c1; });
    trace_entries_part(g.N, q, excl, 1, [&](int col, double v) { h1 += entry_hash(col, v); ++c2; });
    if (h0 != h1 || c0 != c1 + c2) atomicAdd(bad, 1ull);
    if (c2 > 0) atomicAdd(nsplit, 1ull);
  }
}
}  // namespace

int64_t test_split_trace(Problem &P, int64_t *nsplit) {
  AIRT_REQUIRE(P.geo_kind != GEO_NONE && P.geo_kind != GEO_SPHERE, "the problem has no straight-ray geometry");
  cudaStream_t s = P.stream;
  DevBuf<unsigned long long> c;
  c.ensure(2);
  AIRT_CHECK_CUDA(cudaMemsetAsync(c.p, 0, 2 * sizeof(unsigned long long), s));
  k_test_split<<<grid_for(P.m, 128, 16), 128, 0, s>>>(P.geom(), P.m, excl_of(P), c.p, c.p + 1);
  AIRT_LAUNCH_CHECK();
  unsigned long long hc[2] = {0, 0};
  AIRT_CHECK_CUDA(cudaMemcpyAsync(hc, c.p, sizeof(hc), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  if (nsplit) *nsplit = (int64_t)hc[1];
  return (int64_t)hc[0];
}

// Matrix-free pieces of the SIRT iteration (used by sirt.cu).
void mf_backproject_f32(Problem &P, const float *u, double *g64, const int *stop_flag) {
  cudaStream_t s = P.stream;
  if (P.par_ok) {
    par_backproject<float>(P, u, g64, stop_flag);
    return;
  }
  AIRT_CHECK_CUDA(cudaMemsetAsync(P.mf_umax.p, 0, sizeof(unsigned long long), s));
  k_absmax<<<grid_for(P.m, 256), 256, 0, s>>>(P.m, nullptr, u, P.mf_umax.p, stop_flag);
  if (straight(P)) {
    dda_adjoint<float>(P, u, g64, P.mf_umax.p, stop_flag);
    return;
  }
  AIRT_CHECK_CUDA(cudaMemsetAsync(g64, 0, P.n * sizeof(double), s));
  k_mf_adjoint_fx<float><<<grid_for(P.m, 64, 32), 64, 0, s>>>(
      P.geom(), P.m, excl_of(P), u, reinterpret_cast<long long *>(g64), P.mf_kbound, P.mf_umax.p,
      stop_flag);
  k_fx_to_f64<<<grid_for(P.n, 256), 256, 0, s>>>(P.n, g64, P.mf_kbound, P.mf_umax.p, stop_flag);
  AIRT_LAUNCH_CHECK();
}

}  // namespace airt

// All iterations of a small stored problem in one launch.
//
// At a few megabytes of matrix an iteration of launched kernels is latency:
// two launches and, in each product, the chain row pointer -> entries ->
// gather -> sum (12 us per iteration at N = 64, 30 angles, where the bytes
// take less than 1 us).  Here one CTA per SM stays for the whole solve.  A
// group of lanes owns the same rows and columns in every iteration and keeps
// the first kResident 16-byte vectors of its first segment per lane (values
// and indices, both directions) in registers, so that of the chain only the
// gather and the sum remain between two grid barriers; what does not fit is
// read from L2 again.  The stopping rule needs no launch either: every CTA
// adds the CTAs' partial sums in the same order and takes the same decision
// while the gathers of the next update are in flight.
//
// The grid barrier is a counter that every CTA raises and waits on; the
// launch is cooperative, so all CTAs are resident.  Each wait is bounded: on
// expiry the kernel raises the error flag, every CTA leaves, and the host
// reports AIRT_ERR_TIMEOUT.
#pragma once

#include "common.cuh"

namespace airt {

// Cycle budget of a wait, and the test hook that makes one run out (art.cu).
extern long long g_wait_budget;
extern int g_inject_stall;

// One direction of the matrix: segments ptr[i]..ptr[i+1] of idx and val, L
// lanes per segment.
struct PersistDir {
  int nseg;
  const int64_t *ptr;
  const int *idx;
  const float *val;
  int L;
};

// Lanes per segment for `threads` threads: the fewest vector loads in a row per
// lane, where a segment's fixed part (bounds, reduction, epilogue) counts as
// three.
inline int persist_lanes(int64_t nnz, int64_t nseg, int64_t threads) {
  const double avg = nseg ? (double)nnz / (double)nseg : 0.0;
  int best = 2;
  double cost = INFINITY;
  for (int L = 2; L <= 32; L *= 2) {
    const double c = std::ceil((double)nseg * L / (double)threads) * (avg / (4.0 * L) + 3.0);
    if (c < cost) {
      cost = c;
      best = L;
    }
  }
  return best;
}

// The resident part of a lane's first segment: vectors v, v + L, ... of the
// aligned groups that overlap it, a mask bit per element inside the segment,
// and where the rest of the segment's vectors starts.
template <int R>
struct PersistSeg {
  float4 f[R > 0 ? R : 1];
  int4 c[R > 0 ? R : 1];
  unsigned mask;
  int v, ve;     // next vector of this lane and end, relative to base
  int64_t base;  // first vector of the segment
  int lo, hi;    // first and last + 1 element of the segment, relative to 4*base
};

template <int R>
__device__ __forceinline__ PersistSeg<R> persist_load(const PersistDir &d, int seg, int lane) {
  PersistSeg<R> s;
  s.mask = 0;
  int64_t q0 = 0, q1 = 0;
  if (seg < d.nseg) {
    q0 = __ldg(d.ptr + seg);
    q1 = __ldg(d.ptr + seg + 1);
  }
  s.base = q0 >> 2;
  s.lo = (int)(q0 - 4 * s.base);
  s.hi = (int)(q1 - 4 * s.base);
  s.ve = q1 > q0 ? (s.hi + 3) >> 2 : 0;
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int v = lane + u * d.L;
    s.f[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    s.c[u] = make_int4(0, 0, 0, 0);
    if (v < s.ve) {
      s.f[u] = __ldg(reinterpret_cast<const float4 *>(d.val) + s.base + v);
      const int4 c = __ldg(reinterpret_cast<const int4 *>(d.idx) + s.base + v);
      const int e = 4 * v;
      unsigned k = 0;
      if (e >= s.lo && e < s.hi) { k |= 1u; s.c[u].x = c.x; }
      if (e + 1 >= s.lo && e + 1 < s.hi) { k |= 2u; s.c[u].y = c.y; }
      if (e + 2 >= s.lo && e + 2 < s.hi) { k |= 4u; s.c[u].z = c.z; }
      if (e + 3 >= s.lo && e + 3 < s.hi) { k |= 8u; s.c[u].w = c.w; }
      s.mask |= k << (4 * u);
    }
  }
  s.v = lane + R * d.L;
  return s;
}

// A copy of a loop-invariant register that the compiler takes to change: it
// keeps values derived from the resident matrix (FP64 copies, addresses) from
// being held beside it, which spilled 370 bytes at 128 registers.
__device__ __forceinline__ float fresh(float v) {
  asm volatile("" : "+f"(v));
  return v;
}
__device__ __forceinline__ int fresh(int v) {
  asm volatile("" : "+r"(v));
  return v;
}

// Sum over the lane's own elements of a resident segment; x is written by
// other CTAs between barriers, so it is read with plain loads.
template <int R>
__device__ __forceinline__ double persist_dot(const PersistDir &d, const PersistSeg<R> &s, const float *x) {
  float4 g[R > 0 ? R : 1];
#pragma unroll
  for (int u = 0; u < R; ++u)
    if (s.mask >> (4 * u) & 15u) g[u] = make_float4(x[fresh(s.c[u].x)], x[fresh(s.c[u].y)], x[fresh(s.c[u].z)], x[fresh(s.c[u].w)]);
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
#pragma unroll
  for (int u = 0; u < R; ++u) {
    if (s.mask >> (4 * u) & 1u) a0 = fma((double)fresh(s.f[u].x), (double)g[u].x, a0);
    if (s.mask >> (4 * u) & 2u) a1 = fma((double)fresh(s.f[u].y), (double)g[u].y, a1);
    if (s.mask >> (4 * u) & 4u) a2 = fma((double)fresh(s.f[u].z), (double)g[u].z, a2);
    if (s.mask >> (4 * u) & 8u) a3 = fma((double)fresh(s.f[u].w), (double)g[u].w, a3);
  }
#pragma unroll 1
  for (int v = s.v; v < s.ve; v += d.L) {
    const float4 f = __ldg(reinterpret_cast<const float4 *>(d.val) + s.base + v);
    const int4 c = __ldg(reinterpret_cast<const int4 *>(d.idx) + s.base + v);
    const int e = 4 * v;  // v > 0, so only the segment's end can cut the vector
    a0 = fma((double)f.x, (double)x[c.x], a0);
    if (e + 1 < s.hi) a1 = fma((double)f.y, (double)x[c.y], a1);
    if (e + 2 < s.hi) a2 = fma((double)f.z, (double)x[c.z], a2);
    if (e + 3 < s.hi) a3 = fma((double)f.w, (double)x[c.w], a3);
  }
  return (a0 + a1) + (a2 + a3);
}

// The same for a segment that is read again in every iteration.
template <int AHEAD>
__device__ __forceinline__ double persist_dot_again(const PersistDir &d, int seg, int lane, const float *x) {
  int64_t q0 = 0, q1 = 0;
  if (seg < d.nseg) {
    q0 = __ldg(d.ptr + seg);
    q1 = __ldg(d.ptr + seg + 1);
  }
  const int64_t ve = q1 > q0 ? (q1 + 3) >> 2 : 0;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  auto masked = [&](int64_t v) {
    const float4 f = __ldg(reinterpret_cast<const float4 *>(d.val) + v);
    const int4 c = __ldg(reinterpret_cast<const int4 *>(d.idx) + v);
    const int64_t e = v << 2;
    if (e >= q0 && e < q1) a0 = fma((double)f.x, (double)x[c.x], a0);
    if (e + 1 >= q0 && e + 1 < q1) a1 = fma((double)f.y, (double)x[c.y], a1);
    if (e + 2 >= q0 && e + 2 < q1) a2 = fma((double)f.z, (double)x[c.z], a2);
    if (e + 3 >= q0 && e + 3 < q1) a3 = fma((double)f.w, (double)x[c.w], a3);
  };
  // the vectors cut by the segment's ends, then the others AHEAD at a time
  const int64_t vb = (q0 + 3) >> 2, vl = q1 >> 2;
  if (lane == 0 && vb > (q0 >> 2) && q1 > q0) masked(q0 >> 2);
  if (lane == d.L - 1 && vl >= vb && ve > vl) masked(vl);
  int64_t v = vb + lane;
  for (; v + (AHEAD - 1) * d.L < vl; v += AHEAD * d.L) {
    float4 f[AHEAD];
    int4 c[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      f[u] = __ldg(reinterpret_cast<const float4 *>(d.val) + v + u * d.L);
      c[u] = __ldg(reinterpret_cast<const int4 *>(d.idx) + v + u * d.L);
    }
    float4 g[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) g[u] = make_float4(x[c[u].x], x[c[u].y], x[c[u].z], x[c[u].w]);
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      a0 = fma((double)f[u].x, (double)g[u].x, a0);
      a1 = fma((double)f[u].y, (double)g[u].y, a1);
      a2 = fma((double)f[u].z, (double)g[u].z, a2);
      a3 = fma((double)f[u].w, (double)g[u].w, a3);
    }
  }
#pragma unroll 1
  for (; v < vl; v += d.L) {
    const float4 f = __ldg(reinterpret_cast<const float4 *>(d.val) + v);
    const int4 c = __ldg(reinterpret_cast<const int4 *>(d.idx) + v);
    a0 = fma((double)f.x, (double)x[c.x], a0);
    a1 = fma((double)f.y, (double)x[c.y], a1);
    a2 = fma((double)f.z, (double)x[c.z], a2);
    a3 = fma((double)f.w, (double)x[c.w], a3);
  }
  return (a0 + a1) + (a2 + a3);
}

__device__ __forceinline__ double persist_group_sum(double v, int L) {
  for (int o = L >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Raises the counter and waits until it has reached `target`; thread 0 runs
// first() after the CTA's other threads have arrived and before it raises the
// counter.  Returns false (in every thread) when a wait ran out, here or
// elsewhere.
template <class First>
__device__ __forceinline__ bool persist_barrier(unsigned *count, unsigned target, int *err, long long budget,
                                                First &&first) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    first();
    // release and acquire on the counter order the CTAs' other accesses
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    const long long t0 = clock64();
    int good = 1;
    for (unsigned n = 1;; ++n) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
      if (v >= target) break;
      if (n % 64) continue;  // look at the flag and the clock now and then
      if (*(volatile int *)err) {
        good = 0;
        break;
      }
      if (clock64() - t0 > budget) {
        atomicExch(err, 1);
        good = 0;
        break;
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

}  // namespace airt

// All iterations of a small stored problem in one launch.
//
// At a few megabytes of matrix an iteration of launched kernels is latency:
// two launches and, in each product, the chain row pointer -> entries ->
// gather -> sum (12 us per iteration at N = 64, 30 angles, where the bytes
// take less than 1 us).  Here one CTA per SM stays for the whole solve.  A
// group of threads owns the same rows and columns in every iteration and keeps
// the first entries of its first segment per thread (values and indices, both
// directions) in registers, so that of the chain only the gather and the sum
// remain between two grid barriers; what does not fit is read from L2 again.
// The stopping rule needs no launch either: every CTA adds the CTAs' partial
// sums in the same order and takes the same decision while the gathers of the
// next update are in flight.
//
// Every sum is taken in the order of the launched kernels
// (for_each_segment_vpre of spmv.cuh): L lanes per segment, four accumulators
// per lane, one for each element of the 16-byte vectors.  An FP64 sum in
// another order differs in its last bit, which flips the FP32 rounding of x or
// M.*r now and then: 5e-10 of x after 1,500 iterations.  More threads than L
// lanes come from the accumulators: C of the four per thread.
//
// The grid barrier is a counter that every CTA raises and waits on; the
// launch is cooperative, so all CTAs are resident.  Each wait is bounded: on
// expiry the kernel raises the error flag, every CTA leaves, and the host
// reports AIRT_ERR_TIMEOUT.
#pragma once

#include "common.cuh"
#include "spmv.cuh"

namespace airt {

// Cycle budget of a wait, and the test hook that makes one run out (art.cu).
extern long long g_wait_budget;
extern int g_inject_stall;

// One direction of the matrix: segments ptr[i]..ptr[i+1] of idx and val (fewer
// than 2^30 of them and of nonzeros), L lanes of S threads per segment; thread
// `sub` of a lane has the accumulators of the vector elements sub*C .. sub*C + C-1.
struct PersistDir {
  int nseg;
  const int64_t *ptr;
  const int *idx;
  const float *val;
  int L, C, S, T;  // S = 4 / C, T = L * S threads per segment
};

// The split for `threads` threads: L as the launched kernels have it, and the
// C with the fewest vectors' worth of loads in a row per thread, where a
// segment's fixed part (bounds, reduction, epilogue) counts as three.
inline void persist_split(PersistDir &d, int64_t nnz, int64_t threads) {
  const double avg = d.nseg ? (double)nnz / (double)d.nseg : 0.0;
  d.L = vec_lanes_for(nnz, d.nseg);
  double cost = INFINITY;
  for (int C = 4; C >= 1; C /= 2) {
    const int T = d.L * 4 / C;
    const double c = std::ceil((double)d.nseg * T / (double)threads) * (avg / (4.0 * T) + 3.0);
    if (c >= cost) continue;
    cost = c;
    d.C = C;
    d.S = 4 / C;
    d.T = T;
  }
}

// Where a thread's part of a segment lies: nonzeros [q0, q1), whole vectors
// [qa, qb) of them; the others are added first, those before qa to the first
// accumulator, those from qb on to the second.
struct PersistPart {
  int q0, q1, qa, qb, lane, sub;
};

__device__ __forceinline__ PersistPart persist_part(const PersistDir &d, int seg, int t) {
  PersistPart p{0, 0, 0, 0, t / d.S, t % d.S};
  if (seg < d.nseg) {
    p.q0 = (int)__ldg(d.ptr + seg);
    p.q1 = (int)__ldg(d.ptr + seg + 1);
  }
  p.qa = min((p.q0 + 3) & ~3, p.q1);
  p.qb = max(p.q1 & ~3, p.qa);
  return p;
}

// The resident part of a thread's first segment (L > 2, so that a thread has
// at most one element before the whole vectors and one after them): the
// element before, the one after, the first R of the vectors', and where the
// rest starts.
template <int C, int R>
struct PersistSeg {
  float f[R > 0 ? R : 1], fe[2];
  int c[R > 0 ? R : 1], ce[2];
  int have;    // whole vectors held
  bool on[2];  // the element before, the one after
  int v, ve;   // next vector of this lane and end
  int sub;
};

template <int C, int R>
__device__ __forceinline__ PersistSeg<C, R> persist_load(const PersistDir &d, int seg, int t) {
  const PersistPart p = persist_part(d, seg, t);
  PersistSeg<C, R> s;
  s.sub = p.sub;
  const int h = p.q0 + p.lane, g = p.qb + p.lane;
  s.on[0] = p.sub == 0 && h < p.qa;
  s.on[1] = p.sub == (C == 1 ? 1 : 0) && g < p.q1;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    s.fe[i] = s.on[i] ? __ldg(d.val + (i ? g : h)) : 0.f;
    s.ce[i] = s.on[i] ? __ldg(d.idx + (i ? g : h)) : 0;
  }
  const int v0 = (p.qa >> 2) + p.lane;
  s.ve = p.qb >> 2;
  s.have = min(R / C, max(0, (s.ve - v0 + d.L - 1) / d.L));
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int u = i / C, q = 4 * (v0 + u * d.L) + p.sub * C + i % C;
    s.f[i] = u < s.have ? __ldg(d.val + q) : 0.f;
    s.c[i] = u < s.have ? __ldg(d.idx + q) : 0;
  }
  s.v = v0 + R / C * d.L;
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

// Adds vectors v, v + L, .. < ve of the thread's C accumulators to a[0..C),
// AHEAD vectors in flight; x is written by other CTAs between barriers, so it
// is read with plain loads.
template <int C, int AHEAD>
__device__ __forceinline__ void persist_vectors(const PersistDir &d, int v, int ve, int sub, const float *x,
                                                double *a) {
  auto load = [&](int w, float *f, int *c) {
    const float *fp = d.val + 4 * w + sub * C;
    const int *cp = d.idx + 4 * w + sub * C;
    if (C == 4) {
      const float4 f4 = __ldg(reinterpret_cast<const float4 *>(fp));
      const int4 c4 = __ldg(reinterpret_cast<const int4 *>(cp));
      f[0] = f4.x, f[1] = f4.y, f[2] = f4.z, f[3] = f4.w;
      c[0] = c4.x, c[1] = c4.y, c[2] = c4.z, c[3] = c4.w;
    } else if (C == 2) {
      const float2 f2 = __ldg(reinterpret_cast<const float2 *>(fp));
      const int2 c2 = __ldg(reinterpret_cast<const int2 *>(cp));
      f[0] = f2.x, f[1] = f2.y;
      c[0] = c2.x, c[1] = c2.y;
    } else {
      f[0] = __ldg(fp);
      c[0] = __ldg(cp);
    }
  };
#pragma unroll 1
  for (; v + (AHEAD - 1) * d.L < ve; v += AHEAD * d.L) {
    float f[AHEAD][C], g[AHEAD][C];
    int c[AHEAD][C];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) load(v + u * d.L, f[u], c[u]);
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
#pragma unroll
      for (int k = 0; k < C; ++k) g[u][k] = x[c[u][k]];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
#pragma unroll
      for (int k = 0; k < C; ++k) a[k] = fma((double)f[u][k], (double)g[u][k], a[k]);
  }
  if (AHEAD > 1)
#pragma unroll 1
    for (; v < ve; v += d.L) {
      float f[C];
      int c[C];
      load(v, f, c);
#pragma unroll
      for (int k = 0; k < C; ++k) a[k] = fma((double)f[k], (double)x[c[k]], a[k]);
    }
}

template <int C>
__device__ __forceinline__ double persist_fold(const double *a) {
  return C == 4 ? (a[0] + a[1 % C]) + (a[2 % C] + a[3 % C]) : C == 2 ? a[0] + a[1 % C] : a[0];
}

// The thread's part of the sum over a resident segment.
template <int C, int R>
__device__ __forceinline__ double persist_dot(const PersistDir &d, const PersistSeg<C, R> &s, const float *x) {
  float g[R > 0 ? R : 1], ge[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (s.on[i]) ge[i] = x[fresh(s.ce[i])];
#pragma unroll
  for (int i = 0; i < R; ++i)
    if (i / C < s.have) g[i] = x[fresh(s.c[i])];
  double a[C] = {};
  if (s.on[0]) a[0] = fma((double)fresh(s.fe[0]), (double)ge[0], a[0]);
  if (s.on[1]) a[1 % C] = fma((double)fresh(s.fe[1]), (double)ge[1], a[1 % C]);
#pragma unroll
  for (int i = 0; i < R; ++i)
    if (i / C < s.have) a[i % C] = fma((double)fresh(s.f[i]), (double)g[i], a[i % C]);
  persist_vectors<C, 1>(d, s.v, s.ve, s.sub, x, a);
  return persist_fold<C>(a);
}

// The same for a segment that is read again in every iteration.
template <int C, int AHEAD>
__device__ __forceinline__ double persist_again_c(const PersistDir &d, const PersistPart &p, const float *x) {
  double a[C] = {};
  if (p.sub == 0)
    for (int q = p.q0 + p.lane; q < p.qa; q += d.L) a[0] = fma((double)__ldg(d.val + q), (double)x[__ldg(d.idx + q)], a[0]);
  if (p.sub == (C == 1 ? 1 : 0))
    for (int q = p.qb + p.lane; q < p.q1; q += d.L) {
      double &t = a[C > 1 ? 1 % C : 0];
      t = fma((double)__ldg(d.val + q), (double)x[__ldg(d.idx + q)], t);
    }
  persist_vectors<C, AHEAD>(d, (p.qa >> 2) + p.lane, p.qb >> 2, p.sub, x, a);
  return persist_fold<C>(a);
}

// K: the direction's C, or 0 where the kernel is made for any.
template <int K, int AHEAD>
__device__ __forceinline__ double persist_dot_again(const PersistDir &d, int seg, int t, const float *x) {
  const PersistPart p = persist_part(d, seg, t);
  if (K) return persist_again_c<K ? K : 1, AHEAD>(d, p, x);
  return d.C == 4   ? persist_again_c<4, AHEAD>(d, p, x)
         : d.C == 2 ? persist_again_c<2, AHEAD>(d, p, x)
                    : persist_again_c<1, AHEAD>(d, p, x);
}

// Sum over the threads of a segment: a lane's accumulators, then the lanes.
__device__ __forceinline__ double persist_group_sum(double v, const PersistDir &d) {
  for (int o = 1; o < d.S; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  for (int o = d.T >> 1; o >= d.S; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
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

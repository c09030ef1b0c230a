// CART column-action sweeps on the GPU (cart/cart.m:139-320).
//
// A sweep visits the columns j of its order one after the other.  An
// unflagged column takes the step od = relaxpar * (a_j'*r)/||a_j||^2,
// clipped so that x(j) + od stays in the box, adds it to x(j) and subtracts
// od*a_j from the residual r; it is flagged when, from sweep Kbegin on,
// |od| < THR * max(abs(x)) with x as it was before the step.  A flagged
// column is skipped until randi(Nunflag) no longer exceeds its count.
//
// Every step reads the residual the previous step wrote, which as written is
// one dependent pass over memory per column.  k_cart_block takes that pass
// off the chain.  For a block of 32 consecutive columns of the order the
// products a_j'*r are taken from the residual as it was one block earlier and
// corrected inside the chain by the inner products of the columns:
//   a_j'*r_now = a_j'*r_then - sum_i (a_j'*a_i) od_i
// over the steps i since then, which is the same number up to FP64 rounding.
// One warp runs the chain (lane j of a block: one multiply, the clip, a
// shuffle and a multiply-add per column, no memory); the other warps of the
// CTA apply the previous block's steps to the residual and take the next
// block's products meanwhile.  The plan (CartPlan) holds the inner products
// and every block's entries sorted by row, so that a thread owns a row and
// the residual update needs no atomics.
//
// Bound: the workers' issue slots (9,700 instructions per block on three
// schedulers, 5,000 cycles), then the chain (70 cycles per column after 1,200
// cycles at the head of a block).  Measured per sweep, against one warp that
// walked the columns with the residual in shared memory, or one CTA where it
// did not fit: N = 64, 30 angles 4.5 -> 0.26 ms; N = 128, 60 angles 18.3 ->
// 1.16 ms; N = 256, 60 angles 73.5 -> 4.95 ms; N = 256, 180 angles (residual
// in global memory) 118 -> 26.9 ms.  The plan costs 1-6 ms once per matrix
// and order.
//
// The flags of a sweep do not feed back into it when no column repeats in
// the order, so they are settled after the sweep (k_cart_flags): the maximum
// of abs(x) before step t is the larger of the new values' running maximum
// up to t and the old values' running maximum from t on.  Orders that repeat
// a column take the general sweep, a column per step: one warp with the
// residual in shared memory where it fits there (the next column's index,
// flag, x(j), norm and first entries load during the current step; 1.10 us per
// column at N = 256, 60 angles against 1.46 us for a CTA), otherwise one
// 256-thread CTA (N = 256, 180 angles: 1.74 us per column against 2.06 us for
// a warp).  max(abs(x)) is kept exact without an O(n) scan: the maximum of
// every 256-entry block of |x| in shared memory and the overall maximum in a
// register; a step changes one entry, and a block, or the total, is rescanned
// only when the entry that held its maximum shrank.
#include <cub/device/device_radix_sort.cuh>
#include <cuda_pipeline.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "ncp.cuh"

namespace airt {

namespace {

constexpr int kCartThreads = 256;  // threads of the general sweep
constexpr int kCartBlock = 256;  // entries of x per block maximum
constexpr int kCartPre = 8;      // entries per lane the general sweep loads ahead with the next column
constexpr int kCartSmem = 200 * 1024;  // shared memory of the general sweep at most
constexpr int kCartCols = 32;    // columns per block of the blocked sweep: one per lane of its chain
constexpr int kCartBlockThreads = 768;  // 24 warps: 85 registers a thread (1024: spills, 20 % slower)
constexpr int kCartWorkers = kCartBlockThreads * 3 / 4;  // threads beside the chain's (see k_cart_block)
constexpr int kCartRowBits = 27;  // row field of a sorted entry
constexpr unsigned kCartNoRow = (1u << kCartRowBits) - 1;
// rows whose residual fits in shared memory beside the inner products (192 of
// 227 KB); more rows than that keep it in global memory
constexpr int64_t kCartSharedRows = 24000;

struct CartArgs {
  const int64_t *cp;
  const int *ri;
  const float *cv;
  const double *nrm;  // damped squared column norms
  const int *cols;    // sweep order (0-based)
  int64_t ncols;
  double lam;
  double *x, *r;
  unsigned char *flag;  // F of cart.m
  int *nflag;           // Nflag of cart.m
  int lbk, ubk;
  double lb, ub;
  const double *lbv, *ubv;
  double thr;
  int64_t kbegin, nunflag;
  unsigned long long seed;
  int64_t n, m;
  double *r2;  // ||r||^2 after the sweep
  int *err;    // 1: randi(Nunflag) with Nunflag < 1
};

__host__ __device__ inline unsigned long long splitmix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// randi(N) of the unflagging test of sweep k at column j: 1 + floor(u*N)
// with u = the top 53 bits of splitmix64(seed ^ splitmix64(k << 32 | j)).
__device__ inline int64_t cart_randi(unsigned long long seed, int64_t k, int j, int64_t N) {
  const unsigned long long key = ((unsigned long long)k << 32) | (unsigned)j;
  const unsigned long long z = splitmix64(seed ^ splitmix64(key));
  const double u = (double)(z >> 11) * 0x1.0p-53;
  return 1 + min((int64_t)floor(u * (double)N), N - 1);
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum / maximum over the CTA, returned to every thread (the same value in
// all of them: each warp folds the per-warp partials in the same order).
__device__ __forceinline__ double cta_allsum(double v, double *sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = (l < kCartThreads / 32) ? sh[l] : 0.0;
  t = warp_sum(t);
  __syncthreads();
  return t;
}

__device__ __forceinline__ double cta_allmax(double v, double *sh) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = (l < kCartThreads / 32) ? sh[l] : 0.0;
  t = warp_max(t);
  __syncthreads();
  return t;
}



// The prefetched part of one step: the column, its start and end, flag,
// x(j), damped norm, and its first kCartPre*32 entries (lane l holds
// entries s0 + l + 32*u).
struct CartCol {
  int j;
  int64_t s0, s1;
  unsigned char f;
  double xj, nrm;
  int ri[kCartPre];
  float cv[kCartPre];
};

__device__ __forceinline__ void cart_load(const CartArgs &a, int64_t t, CartCol &c) {
  const int lane = threadIdx.x;
  c.j = a.cols[t];
  c.s0 = a.cp[c.j];
  c.s1 = a.cp[c.j + 1];
  c.f = a.flag[c.j];
  c.xj = a.x[c.j];
  c.nrm = a.nrm[c.j];
#pragma unroll
  for (int u = 0; u < kCartPre; ++u) {
    const int64_t q = c.s0 + lane + 32 * u;
    c.ri[u] = q < c.s1 ? a.ri[q] : 0;
    c.cv[u] = q < c.s1 ? a.cv[q] : 0.f;
  }
}

// One sweep, one warp (launched as a single 32-thread CTA), with the
// residual copied into shared memory for the sweep and back after it.  Sums
// and maxima use xor shuffles, which leave the same value in every lane.
__global__ void __launch_bounds__(32) k_cart_sweep_warp(CartArgs a, int64_t k) {
  extern __shared__ double smem[];
  const int lane = threadIdx.x;
  const int64_t nb = (a.n + kCartBlock - 1) / kCartBlock;
  double *bmax = smem;  // max |x| of each kCartBlock-entry block
  double *r = smem + ((nb + 1) & ~(int64_t)1);
  for (int64_t i = lane; i < a.m; i += 32) r[i] = a.r[i];
  for (int64_t b = 0; b < nb; ++b) {
    double v = 0.0;
    for (int u = lane; u < kCartBlock; u += 32) {
      const int64_t i = b * kCartBlock + u;
      if (i < a.n) v = fmax(v, fabs(a.x[i]));
    }
    v = warp_max(v);
    if (lane == 0) bmax[b] = v;
  }
  __syncwarp();
  double M = 0.0;
  {
    double v = 0.0;
    for (int64_t b = lane; b < nb; b += 32) v = fmax(v, bmax[b]);
    M = warp_max(v);
  }
  const bool lbon = a.lbk != AIRT_BOUND_NONE, ubon = a.ubk != AIRT_BOUND_NONE;
  CartCol cur, nxt;
  if (a.ncols > 0) cart_load(a, 0, cur);
  int prev = -1;
  for (int64_t t = 0; t < a.ncols; ++t) {
    if (t + 1 < a.ncols) cart_load(a, t + 1, nxt);  // in flight during this step
    const int j = cur.j;
    if (j == prev) {  // the prefetch predates the previous step on the same column
      cur.f = a.flag[j];
      cur.xj = a.x[j];
    }
    if (cur.f) {
      const double mm = M;  // max(abs(xk)) before the step, cart.m:227
      double part = 0.0;
#pragma unroll
      for (int u = 0; u < kCartPre; ++u)
        if (cur.s0 + lane + 32 * u < cur.s1) part = fma((double)cur.cv[u], r[cur.ri[u]], part);
      for (int64_t q = cur.s0 + lane + 32 * kCartPre; q < cur.s1; q += 32)
        part = fma((double)a.cv[q], r[a.ri[q]], part);
      const double dot = warp_sum(part);
      // cart.m:242-278
      double od = __dmul_rn(a.lam, __ddiv_rn(dot, cur.nrm));
      const double xkj = cur.xj;
      if (lbon) {
        const double lo = __dsub_rn(a.lbk == AIRT_BOUND_SCALAR ? a.lb : a.lbv[j], xkj);
        if (od < lo) od = lo;
      }
      if (ubon) {
        const double hi = __dsub_rn(a.ubk == AIRT_BOUND_SCALAR ? a.ub : a.ubv[j], xkj);
        if (od > hi) od = hi;
      }
      const double xn = __dadd_rn(xkj, od);
#pragma unroll
      for (int u = 0; u < kCartPre; ++u)
        if (cur.s0 + lane + 32 * u < cur.s1) {
          const int i = cur.ri[u];
          r[i] = __dsub_rn(r[i], __dmul_rn(od, (double)cur.cv[u]));
        }
      for (int64_t q = cur.s0 + lane + 32 * kCartPre; q < cur.s1; q += 32) {
        const int i = a.ri[q];
        r[i] = __dsub_rn(r[i], __dmul_rn(od, (double)a.cv[q]));
      }
      if (lane == 0) {
        a.x[j] = xn;
        if (k >= a.kbegin && fabs(od) < a.thr * mm) {
          a.flag[j] = 0;
          a.nflag[j] = 1;
        }
      }
      // running maximum of |x|
      const int64_t b = j / kCartBlock;
      const double cur_b = bmax[b], ao = fabs(xkj), an = fabs(xn);
      __syncwarp();  // x(j), r and the flags are written; bmax[b] is read
      double nbv = cur_b;
      if (an >= cur_b) {
        nbv = an;
      } else if (ao == cur_b) {  // the entry that held the block's maximum shrank
        double v = 0.0;
        for (int u = lane; u < kCartBlock; u += 32) {
          const int64_t i = b * kCartBlock + u;
          if (i < a.n) v = fmax(v, fabs(a.x[i]));
        }
        nbv = warp_max(v);
      }
      if (nbv >= M) {
        M = nbv;
      } else if (cur_b == M) {  // the block that held the overall maximum dropped
        if (lane == 0) bmax[b] = nbv;
        __syncwarp();
        double v = 0.0;
        for (int64_t bb = lane; bb < nb; bb += 32) v = fmax(v, bmax[bb]);
        M = warp_max(v);
      }
      __syncwarp();
      if (lane == 0) bmax[b] = nbv;
      __syncwarp();
    } else {
      if (lane == 0) {  // cart.m:281-285
        if (a.nunflag < 1) {
          *a.err = 1;
        } else if (a.nflag[j] < cart_randi(a.seed, k, j, a.nunflag)) {
          a.nflag[j] += 1;
        } else {
          a.flag[j] = 1;
        }
      }
      __syncwarp();
    }
    prev = j;
    cur = nxt;
  }
  double v = 0.0;
  for (int64_t i = lane; i < a.m; i += 32) {
    const double ri = r[i];
    v += ri * ri;
    a.r[i] = ri;
  }
  v = warp_sum(v);
  if (lane == 0) *a.r2 = v;
}

// One sweep by one 256-thread CTA with the residual in global memory (used
// when the residual does not fit in shared memory): every column's entries
// are spread over all threads, with block barriers between the steps.
__global__ void __launch_bounds__(kCartThreads) k_cart_sweep_cta(CartArgs a, int64_t k) {
  extern __shared__ double bmax[];  // max |x| of each kCartBlock-entry block
  __shared__ double sh[kCartThreads / 32];
  const int tid = threadIdx.x;
  const int64_t nb = (a.n + kCartBlock - 1) / kCartBlock;
  for (int64_t b = 0; b < nb; ++b) {
    const int64_t i = b * kCartBlock + tid;
    const double v = cta_allmax(i < a.n ? fabs(a.x[i]) : 0.0, sh);
    if (tid == 0) bmax[b] = v;
  }
  __syncthreads();
  double M = 0.0;
  {
    double v = 0.0;
    for (int64_t b = tid; b < nb; b += kCartThreads) v = fmax(v, bmax[b]);
    M = cta_allmax(v, sh);
  }
  const bool lbon = a.lbk != AIRT_BOUND_NONE, ubon = a.ubk != AIRT_BOUND_NONE;
  for (int64_t t = 0; t < a.ncols; ++t) {
    const int j = a.cols[t];
    if (a.flag[j]) {
      const double mm = M;  // max(abs(xk)) before the step, cart.m:227
      const int64_t s0 = a.cp[j], s1 = a.cp[j + 1];
      double part = 0.0;
      for (int64_t q = s0 + tid; q < s1; q += kCartThreads)
        part = fma((double)a.cv[q], a.r[a.ri[q]], part);
      const double dot = cta_allsum(part, sh);
      // cart.m:242-278
      double od = __dmul_rn(a.lam, __ddiv_rn(dot, a.nrm[j]));
      const double xkj = a.x[j];
      if (lbon) {
        const double lo = __dsub_rn(a.lbk == AIRT_BOUND_SCALAR ? a.lb : a.lbv[j], xkj);
        if (od < lo) od = lo;
      }
      if (ubon) {
        const double hi = __dsub_rn(a.ubk == AIRT_BOUND_SCALAR ? a.ub : a.ubv[j], xkj);
        if (od > hi) od = hi;
      }
      const double xn = __dadd_rn(xkj, od);
      for (int64_t q = s0 + tid; q < s1; q += kCartThreads) {
        const int i = a.ri[q];
        a.r[i] = __dsub_rn(a.r[i], __dmul_rn(od, (double)a.cv[q]));
      }
      if (tid == 0) {
        a.x[j] = xn;
        if (k >= a.kbegin && fabs(od) < a.thr * mm) {
          a.flag[j] = 0;
          a.nflag[j] = 1;
        }
      }
      // running maximum of |x|
      const int64_t b = j / kCartBlock;
      const double cur = bmax[b], ao = fabs(xkj), an = fabs(xn);
      __syncthreads();  // x(j), r and the flags are written; bmax[b] is read
      double nbv = cur;
      if (an >= cur) {
        nbv = an;
      } else if (ao == cur) {  // the entry that held the block's maximum shrank
        const int64_t i = b * kCartBlock + tid;
        nbv = cta_allmax(i < a.n ? fabs(a.x[i]) : 0.0, sh);
      }
      if (nbv >= M) {
        M = nbv;
      } else if (cur == M) {  // the block that held the overall maximum dropped
        if (tid == 0) bmax[b] = nbv;
        __syncthreads();
        double v = 0.0;
        for (int64_t bb = tid; bb < nb; bb += kCartThreads) v = fmax(v, bmax[bb]);
        M = cta_allmax(v, sh);
      }
      if (tid == 0) bmax[b] = nbv;
      __syncthreads();
    } else {
      if (tid == 0) {  // cart.m:281-285
        if (a.nunflag < 1) {
          *a.err = 1;
        } else if (a.nflag[j] < cart_randi(a.seed, k, j, a.nunflag)) {
          a.nflag[j] += 1;
        } else {
          a.flag[j] = 1;
        }
      }
      __syncthreads();
    }
  }
  double v = 0.0;
  for (int64_t i = tid; i < a.m; i += kCartThreads) v += a.r[i] * a.r[i];
  v = cta_allsum(v, sh);
  if (tid == 0) *a.r2 = v;
}

// Inner products of the columns of block blockIdx.x with each other and with
// those of the block before it: gram[(block*64 + s)*32 + i] = a_i'*a_s, where
// s < 32 are the previous block's columns.  A warp takes column i; its lanes
// hold two of the 64 columns s and follow column i's rows through them (rows
// ascend in every column).
__global__ void __launch_bounds__(1024) k_cart_gram(CartArgs a, double *__restrict__ gram) {
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * kCartCols + i;
  int64_t q0 = 0, q1 = 0;
  if (t < a.ncols) {
    const int j = a.cols[t];
    q0 = a.cp[j];
    q1 = a.cp[j + 1];
  }
  for (int half = 0; half < 2; ++half) {
    const int64_t ts = ((int64_t)blockIdx.x - 1 + half) * kCartCols + lane;
    int64_t p = 0, p1 = 0;
    if (ts >= 0 && ts < a.ncols) {
      const int j = a.cols[ts];
      p = a.cp[j];
      p1 = a.cp[j + 1];
    }
    double acc = 0.0;
    for (int64_t q = q0; q < q1; ++q) {
      const int row = __ldg(a.ri + q);
      const double v = (double)__ldg(a.cv + q);
      while (p < p1 && __ldg(a.ri + p) < row) ++p;
      if (p < p1 && __ldg(a.ri + p) == row) acc = fma(v, (double)__ldg(a.cv + p), acc);
    }
    // lane s of this warp holds G(i, s); the chain reads row s across lanes i
    gram[((int64_t)blockIdx.x * 2 * kCartCols + half * kCartCols + lane) * kCartCols + i] = acc;
  }
}

// Sort key (block, row) and payload (column of the block, value) of every
// entry of the order's columns, one warp per position.
__global__ void k_cart_keys(CartArgs a, const int64_t *__restrict__ off, int rowbits, unsigned *__restrict__ key,
                            unsigned long long *__restrict__ pay) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t t = w; t < a.ncols; t += nw) {
    const int j = a.cols[t];
    const int64_t s0 = a.cp[j], len = a.cp[j + 1] - s0;
    for (int64_t q = lane; q < len; q += 32) {
      key[off[t] + q] = ((unsigned)(t / kCartCols) << rowbits) | (unsigned)a.ri[s0 + q];
      pay[off[t] + q] = ((unsigned long long)(t % kCartCols) << 32) | __float_as_uint(a.cv[s0 + q]);
    }
  }
}

__global__ void k_cart_len(CartArgs a, int64_t *__restrict__ len) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < a.ncols;
       t += (int64_t)gridDim.x * blockDim.x)
    len[t] = a.cp[a.cols[t] + 1] - a.cp[a.cols[t]];
}

__global__ void k_cart_boff(int64_t ncols, int64_t nblocks, const int64_t *__restrict__ off,
                            int64_t *__restrict__ boff) {
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b <= nblocks;
       b += (int64_t)gridDim.x * blockDim.x)
    boff[b] = off[min(b * kCartCols, ncols)];
}

// Second sort key (block, entries of the row in the block) of entries sorted
// by (block, row), and the packed entry.  Rows of one length lie together
// after it, so that most chunks add up short rows only.
__global__ void k_cart_runs(int64_t cnt, int rowbits, const unsigned *__restrict__ key,
                            const unsigned long long *__restrict__ pay, unsigned *__restrict__ key2,
                            unsigned long long *__restrict__ ent) {
  const unsigned rowmask = (unsigned)((1ull << rowbits) - 1);
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < cnt;
       q += (int64_t)gridDim.x * blockDim.x) {
    const unsigned k = key[q];
    int64_t lo = q, hi = q + 1;
    while (lo > 0 && key[lo - 1] == k) --lo;
    while (hi < cnt && key[hi] == k) ++hi;
    key2[q] = (unsigned)((unsigned long long)k >> rowbits) * 64u + (unsigned)(hi - lo);
    ent[q] = (pay[q] & 0xffffffffu) << 32 | (unsigned long long)((k & rowmask) | (unsigned)(pay[q] >> 32) << kCartRowBits);
  }
}

// Cuts a block's sorted entries into chunks of at most 32 that end between
// rows (a row has at most 32 entries in a block), one warp per block.  FILL
// false counts the chunks; true writes them, padded with row kCartNoRow.
template <bool FILL>
__global__ void k_cart_chunks(int64_t nblocks, const int64_t *__restrict__ boff,
                              const unsigned long long *__restrict__ sorted, int64_t *__restrict__ count,
                              const int64_t *__restrict__ cbase, uint2 *__restrict__ ent) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t b = w; b < nblocks; b += nw) {
    const int64_t e1 = boff[b + 1];
    int64_t s = boff[b], c = 0;
    while (s < e1) {
      const int64_t e = s + lane;
      const unsigned long long v = e < e1 ? sorted[e] : 0ull;
      // whether entry e is the last of its row (or the block's)
      const bool last = e < e1 && (e + 1 == e1 || (((unsigned)sorted[e + 1] ^ (unsigned)v) & kCartNoRow));
      const unsigned m = __ballot_sync(0xffffffffu, last);
      const int len = 32 - __clz(m);  // up to the last row end in the window
      if (FILL)
        ent[(cbase[b] + c) * 32 + lane] =
            lane < len ? make_uint2((unsigned)v, (unsigned)(v >> 32)) : make_uint2(kCartNoRow, 0u);
      s += len;
      ++c;
    }
    if (!FILL && lane == 0) count[b] = c;
  }
}

struct CartBlocks {
  int64_t nblocks;
  const int64_t *cbase;
  const uint2 *ent;
  const double *gram;
  double *od;  // the step of every position (0 for skipped columns)
};

__device__ __forceinline__ void cart_worker_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kCartWorkers) : "memory");
}
__device__ __forceinline__ void cart_sync() {
  asm volatile("bar.sync 2, %0;" ::"n"(kCartWorkers + 32) : "memory");
}

// One sweep by one CTA (see the file comment).  While warp 0 runs the chain
// of block b, the workers bring the residual up to block b - 1 and take the
// products of block b + 1 (16 lanes per column).  What they read of the
// matrix is loaded one block ahead, into registers and, for the inner
// products, into shared memory by asynchronous copies.  The workers are the
// warps of the other three SM sub-partitions, so the chain has a scheduler
// and an FP64 pipe to itself.  SMEM: the residual lives in shared memory for
// the sweep (its gathers are scattered: a block's 2,500 entries at N = 256,
// 60 angles take that many L1 cycles, more than the chain).
template <bool SMEM>
__global__ void __launch_bounds__(kCartBlockThreads) k_cart_block(CartArgs a, CartBlocks B) {
  extern __shared__ double2 cart_smem[];
  __shared__ double dots[2][kCartCols], steps[2][kCartCols];
  __shared__ double red[32];
  constexpr int kG = 2 * kCartCols * kCartCols;
  double *const G = reinterpret_cast<double *>(cart_smem);  // [2][64][32]
  double *const r = SMEM ? G + 2 * kG : a.r;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kAhead = 8, kChunks = 6, kWarps = kCartWorkers / 32;
  if (warp > 0 && (warp & 3) == 0) return;
  const int ww = warp - 1 - (warp >> 2), wt = 32 * ww + lane;  // worker warp and thread
  if (SMEM) {
    if (warp > 0)
      for (int64_t i = wt; i < a.m; i += kCartWorkers) r[i] = a.r[i];
    cart_sync();
  }
  if (warp > 0) {
    const int c = wt >> 4, l = wt & 15;
    const bool dotter = c < kCartCols;
    auto fetch_gram = [&](int64_t b) {
      if (b >= B.nblocks) return;
      const double2 *src = reinterpret_cast<const double2 *>(B.gram + b * kG);
      double2 *dst = reinterpret_cast<double2 *>(G + (b & 1) * kG);
      for (int q = wt; q < kG / 2; q += kCartWorkers) __pipeline_memcpy_async(dst + q, src + q, sizeof(double2));
    };
    // r -= steps of a block, a chunk per warp: the products of a row's
    // entries are added across the lanes, the row's first lane owns it
    auto update_chunk = [&](uint2 n, const double *od) {
      const unsigned row = n.x & kCartNoRow;
      const bool in = row != kCartNoRow;
      const unsigned before = __shfl_up_sync(0xffffffffu, row, 1);
      const bool head = in && (lane == 0 || before != row);
      const double rv = head ? r[row] : 0.0;
      double p = (double)__uint_as_float(n.y) * od[n.x >> kCartRowBits];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned k = __shfl_down_sync(0xffffffffu, row, o);
        const bool same = in && lane + o < 32 && k == row;
        if (!__any_sync(0xffffffffu, same)) break;  // rows are runs
        const double q = __shfl_down_sync(0xffffffffu, p, o);
        if (same) p += q;
      }
      if (head) r[row] = rv - p;
    };
    // chunks of this warp in the next block to update: the first kChunks, and
    // where the rest of its `left` chunks lies
    uint2 ent[kChunks];
    const uint2 *rest = B.ent;
    int left = 0;
    int64_t b0 = __ldg(B.cbase), b1 = __ldg(B.cbase + 1);  // of the block to load next
    auto load_chunks = [&](int64_t b) {
      const uint2 *src = B.ent + (b0 + ww) * 32 + lane;
      left = ((int)(b1 - b0) - ww + kWarps - 1) / kWarps;
      b0 = b1;
      if (b + 2 <= B.nblocks) b1 = __ldg(B.cbase + b + 2);
#pragma unroll
      for (int u = 0; u < kChunks; ++u)
        if (u < left) ent[u] = __ldg(src + u * kWarps * 32);
      rest = src + kChunks * kWarps * 32;
    };
    auto update_block = [&](int64_t b) {
      const double *od = steps[b & 1];
#pragma unroll
      for (int u = 0; u < kChunks; ++u)
        if (u < left) update_chunk(ent[u], od);
      for (int u = kChunks; u < left; ++u, rest += kWarps * 32) update_chunk(__ldg(rest), od);
    };
    // products: entries of the next block to take (ri, cv), bounds of the
    // column after it (n0, n1) and the column after that (nc): no load waits
    // for another within a block
    int ri[kAhead];
    float cv[kAhead];
    int have = 0;  // entries of this lane's column from its own on
    const int *pr = a.ri;
    const float *pv = a.cv;
    int64_t n0 = 0, n1 = 0;
    int nc = -1;
    auto load_column = [&](int64_t b) {  // bounds of nc (block b), then nc of block b + 1
      n0 = n1 = 0;
      if (nc >= 0) {
        n0 = __ldg(a.cp + nc);
        n1 = __ldg(a.cp + nc + 1);
      }
      const int64_t t = (b + 1) * kCartCols + c;
      nc = dotter && t < a.ncols ? __ldg(a.cols + t) : -1;
    };
    auto load_entries = [&] {
      have = (int)(n1 - n0) - l;
      pr = a.ri + n0 + l;
      pv = a.cv + n0 + l;
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (16 * u < have) {
          ri[u] = __ldg(pr + 16 * u);
          cv[u] = __ldg(pv + 16 * u);
        }
    };
    auto take_dots = [&](int64_t b) {
      double p0 = 0.0, p1 = 0.0;
#pragma unroll
      for (int u = 0; u < kAhead; u += 2) {
        if (16 * u < have) p0 = fma((double)cv[u], r[ri[u]], p0);
        if (16 * (u + 1) < have) p1 = fma((double)cv[u + 1], r[ri[u + 1]], p1);
      }
      for (int q = 16 * kAhead; q < have; q += 16) p0 = fma((double)__ldg(pv + q), r[__ldg(pr + q)], p0);
      p0 += p1;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) p0 += __shfl_xor_sync(0xffffffffu, p0, o, 16);
      if (dotter && l == 0) dots[b & 1][c] = p0;
    };
    fetch_gram(0);
    load_column(-1);
    load_column(0);
    load_entries();
    load_column(1);
    take_dots(0);
    load_entries();
    load_column(2);
    __pipeline_commit();
    __pipeline_wait_prior(0);
    cart_sync();
    for (int64_t b = 0; b < B.nblocks; ++b) {
      fetch_gram(b + 1);
      __pipeline_commit();
      if (b > 0) update_block(b - 1);
      load_chunks(b);
      cart_worker_sync();
      if (dotter) {
        take_dots(b + 1);
        load_entries();
        load_column(b + 3);
      }
      __pipeline_wait_prior(0);
      cart_sync();
    }
    update_block(B.nblocks - 1);
  } else {
    const bool lbon = a.lbk != AIRT_BOUND_NONE, ubon = a.ubk != AIRT_BOUND_NONE;
    // the columns of the next block (nj and their data) and of the block after
    // it (nj2), loaded during the current one
    int nj = -1, nj2 = -1;
    double nx = 0.0, nn = 1.0, nlo = 0.0, nhi = 0.0;
    unsigned char non = 0;
    auto load_next = [&](int64_t b) {  // data of block b, columns of block b + 1
      nj = nj2;
      if (nj >= 0) {
        nx = a.x[nj];
        nn = __ldg(a.nrm + nj);
        non = a.flag[nj];
        nlo = a.lbk == AIRT_BOUND_VECTOR ? __ldg(a.lbv + nj) : a.lb;
        nhi = a.ubk == AIRT_BOUND_VECTOR ? __ldg(a.ubv + nj) : a.ub;
      }
      const int64_t t = (b + 1) * kCartCols + lane;
      nj2 = t < a.ncols ? __ldg(a.cols + t) : -1;
    };
    load_next(-1);
    load_next(0);
    cart_sync();
    for (int64_t b = 0; b < B.nblocks; ++b) {
      const int j = nj;
      const double xj = nx;
      // skipped columns and lanes past the end: a step clipped to [0, 0]
      const bool on = j >= 0 && non;
      const double c = on ? a.lam / nn : 0.0;
      const double hi = on ? (ubon ? __dsub_rn(nhi, xj) : INFINITY) : 0.0;
      double lo = on ? (lbon ? __dsub_rn(nlo, xj) : -INFINITY) : 0.0;
      if (lo > hi) lo = hi;  // the upper bound is applied last
      load_next(b + 1);
      const double *Gb = G + (b & 1) * kG + lane;
      double d = dots[b & 1][lane];
      if (b > 0) {  // the previous block's steps are not in the residual yet
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        const double *od = steps[(b - 1) & 1];
#pragma unroll
        for (int s = 0; s < kCartCols; s += 4) {
          s0 = fma(Gb[s * kCartCols], od[s], s0);
          s1 = fma(Gb[(s + 1) * kCartCols], od[s + 1], s1);
          s2 = fma(Gb[(s + 2) * kCartCols], od[s + 2], s2);
          s3 = fma(Gb[(s + 3) * kCartCols], od[s + 3], s3);
        }
        d -= (s0 + s1) + (s2 + s3);
      }
      // e = relaxpar * (a_j'*r)/||a_j||^2 (cart.m:242-278), kept scaled so that
      // a step of the chain is the clip, the shuffle and one multiply-add
      double e = d * c, mine = 0.0;
#pragma unroll
      for (int i = 0; i < kCartCols; ++i) {
        const double g = -c * Gb[(kCartCols + i) * kCartCols];
        const bool below = e < lo, above = e > hi;
        double od = below ? lo : e;
        od = above ? hi : od;
        if (lane == i) mine = od;
        e = fma(g, __shfl_sync(0xffffffffu, od, i), e);
      }
      if (!on) mine = 0.0;
      steps[b & 1][lane] = mine;
      if (j >= 0) {
        if (on) a.x[j] = __dadd_rn(xj, mine);
        B.od[b * kCartCols + lane] = mine;
      }
      cart_sync();
    }
  }
  cart_sync();
  double v = 0.0;
  if (warp > 0) {
    for (int64_t i = wt; i < a.m; i += kCartWorkers) {
      const double ri = r[i];
      v = fma(ri, ri, v);
      if (SMEM) a.r[i] = ri;
    }
    v = warp_sum(v);
    if (lane == 0) red[ww] = v;
  }
  cart_sync();
  if (warp == 0) {
    v = warp_sum(lane < kWarps ? red[lane] : 0.0);
    if (lane == 0) *a.r2 = v;
  }
}

// Inclusive running maximum over the CTA's threads in thread order.
__device__ __forceinline__ double cta_scan_max(double v, double *sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = fmax(v, u);
  }
  if (lane == 31) sh[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; ++w) v = fmax(v, sh[w]);
  __syncthreads();
  return v;
}

// Flags of a sweep over an order without repeats, one CTA: mm of step t
// (cart.m:227) is max(abs(x)) with the new values of the positions before t
// and the old values of the others.  tail[t]: work space, the running maximum
// of the old values from t on.
__global__ void __launch_bounds__(1024)
    k_cart_flags(CartArgs a, int64_t k, const double *__restrict__ xold, const double *__restrict__ od,
                 const unsigned char *__restrict__ inorder, double *__restrict__ tail) {
  __shared__ double sh[32];
  const int tid = threadIdx.x;
  const int64_t per = (a.ncols + 1023) / 1024;
  // columns outside the order
  double v = 0.0;
  for (int64_t j = tid; j < a.n; j += 1024)
    if (!inorder[j]) v = fmax(v, fabs(a.x[j]));
  v = warp_max(v);
  if ((tid & 31) == 0) sh[tid >> 5] = v;
  __syncthreads();
  double rest = 0.0;
  for (int w = 0; w < 32; ++w) rest = fmax(rest, sh[w]);
  __syncthreads();
  // old values from t on: thread tid takes the tid-th chunk from the end
  const int64_t hi = a.ncols - (int64_t)tid * per, lo = max(hi - per, (int64_t)0);
  double own = 0.0;
  for (int64_t t = hi - 1; t >= lo; --t) own = fmax(own, fabs(xold[a.cols[t]]));
  double after = cta_scan_max(own, sh);  // own chunk and all later positions
  {
    const double prev = __shfl_up_sync(0xffffffffu, after, 1);
    __shared__ double edge[32];
    if ((tid & 31) == 31) edge[tid >> 5] = after;
    __syncthreads();
    double run = (tid & 31) ? prev : (tid ? edge[(tid >> 5) - 1] : 0.0);
    for (int64_t t = hi - 1; t >= lo; --t) {
      run = fmax(run, fabs(xold[a.cols[t]]));
      tail[t] = run;
    }
  }
  __syncthreads();
  // new values before t
  const int64_t b0 = (int64_t)tid * per, b1 = min(b0 + per, a.ncols);
  own = 0.0;
  for (int64_t t = b0; t < b1; ++t) own = fmax(own, fabs(a.x[a.cols[t]]));
  const double incl = cta_scan_max(own, sh);
  __shared__ double edge2[32];
  if ((tid & 31) == 31) edge2[tid >> 5] = incl;
  const double prev = __shfl_up_sync(0xffffffffu, incl, 1);
  __syncthreads();
  double run = (tid & 31) ? prev : (tid ? edge2[(tid >> 5) - 1] : 0.0);
  for (int64_t t = b0; t < b1; ++t) {
    const int j = a.cols[t];
    const double mm = fmax(rest, fmax(run, tail[t]));
    run = fmax(run, fabs(a.x[j]));
    if (a.flag[j]) {
      if (k >= a.kbegin && fabs(od[t]) < a.thr * mm) {
        a.flag[j] = 0;
        a.nflag[j] = 1;
      }
    } else if (a.nunflag < 1) {  // cart.m:281-285
      *a.err = 1;
    } else if (a.nflag[j] < cart_randi(a.seed, k, j, a.nunflag)) {
      a.nflag[j] += 1;
    } else {
      a.flag[j] = 1;
    }
  }
}

// Squared norms of the CSC columns (cart.m:155-171).
__global__ void k_colnorm2(int64_t n, const int64_t *__restrict__ cp, const float *__restrict__ cv,
                           double *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t j = w; j < n; j += nw) {
    double s = 0;
    for (int64_t q = cp[j] + lane; q < cp[j + 1]; q += 32) {
      const double v = (double)cv[q];
      s += v * v;
    }
    s = warp_sum(s);
    if (lane == 0) out[j] = s;
  }
}

__global__ void k_sub_from(int64_t m, const double *__restrict__ b, double *__restrict__ r) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x)
    r[i] = b[i] - r[i];
}

__global__ void k_sumsq(int64_t m, const double *__restrict__ r, double *__restrict__ out) {
  double v = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x)
    v += r[i] * r[i];
  v = block_sum<256>(v);
  if (threadIdx.x == 0) atomicAdd(out, v);
}

int bits_for(int64_t count) {  // bits that hold 0..count-1
  int b = 1;
  while (b < 62 && (1ll << b) < count) ++b;
  return b;
}

// Plan of the blocked sweep (CartPlan) for a.cols = P.cart_plan.cols.
void build_plan(Problem &P, CartArgs a, cudaStream_t s) {
  CartPlan &C = P.cart_plan;
  C.nblocks = (a.ncols + kCartCols - 1) / kCartCols;
  DevBuf<int64_t> len, off;
  len.ensure(a.ncols);
  off.ensure(a.ncols + 1);
  k_cart_len<<<grid_for(a.ncols, 256), 256, 0, s>>>(a, len.p);
  AIRT_LAUNCH_CHECK();
  exclusive_scan_i64(len.p, off.p, a.ncols, s);
  int64_t cnt = 0;
  AIRT_CHECK_CUDA(cudaMemcpyAsync(&cnt, off.p + a.ncols, sizeof(cnt), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  DevBuf<int64_t> boff, nch;
  boff.ensure(C.nblocks + 1);
  nch.ensure(C.nblocks);
  k_cart_boff<<<grid_for(C.nblocks + 1, 256), 256, 0, s>>>(a.ncols, C.nblocks, off.p, boff.p);
  C.gram.ensure((size_t)C.nblocks * 2 * kCartCols * kCartCols);
  k_cart_gram<<<(unsigned)C.nblocks, 1024, 0, s>>>(a, C.gram.p);
  AIRT_LAUNCH_CHECK();
  const int rowbits = bits_for(a.m), bits = rowbits + bits_for(C.nblocks);
  DevBuf<unsigned> key, key2;
  DevBuf<unsigned long long> pay, pay2;
  DevBuf<unsigned char> tmp;
  key.ensure(cnt);
  key2.ensure(cnt);
  pay.ensure(cnt);
  pay2.ensure(cnt);
  k_cart_keys<<<grid_for(a.ncols * 32, 256), 256, 0, s>>>(a, off.p, rowbits, key.p, pay.p);
  AIRT_LAUNCH_CHECK();
  size_t need = 0;
  AIRT_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, need, key.p, key2.p, pay.p, pay2.p, (int)cnt, 0, bits, s));
  tmp.ensure(need);
  AIRT_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, need, key.p, key2.p, pay.p, pay2.p, (int)cnt, 0, bits, s));
  k_cart_runs<<<grid_for(cnt, 256), 256, 0, s>>>(cnt, rowbits, key2.p, pay2.p, key.p, pay.p);
  AIRT_LAUNCH_CHECK();
  const int bits2 = 6 + bits_for(C.nblocks);
  AIRT_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, need, key.p, key2.p, pay.p, pay2.p, (int)cnt, 0, bits2, s));
  tmp.ensure(need);
  AIRT_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, need, key.p, key2.p, pay.p, pay2.p, (int)cnt, 0, bits2, s));
  const unsigned gc = grid_for(C.nblocks * 32, 128);
  k_cart_chunks<false><<<gc, 128, 0, s>>>(C.nblocks, boff.p, pay2.p, nch.p, nullptr, nullptr);
  AIRT_LAUNCH_CHECK();
  C.cbase.ensure(C.nblocks + 1);
  exclusive_scan_i64(nch.p, C.cbase.p, C.nblocks, s);
  int64_t chunks = 0;
  AIRT_CHECK_CUDA(cudaMemcpyAsync(&chunks, C.cbase.p + C.nblocks, sizeof(chunks), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  C.ent.ensure(chunks * 32);
  k_cart_chunks<true><<<gc, 128, 0, s>>>(C.nblocks, boff.p, pay2.p, nullptr, C.cbase.p, C.ent.p);
  AIRT_LAUNCH_CHECK();
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));  // the work space is freed on return
}

}  // namespace

void run_cart(Problem &P, const airt_cart_opts &o, const double *d_b, const double *d_x0,
              const int64_t *K, int64_t nK, double *d_X, double *resn_host, airt_info *info) {
  cudaStream_t s = P.stream;
  const int64_t m = P.m, n = P.n;
  AIRT_REQUIRE(!P.matrix_free, "CART needs the stored matrix (column access)");
  AIRT_REQUIRE(nK >= 1 && K, "Max no. of iterations must ALWAYS be specified.");
  for (int64_t l = 1; l < nK; ++l)
    AIRT_REQUIRE(K[l] > K[l - 1], "Elements of K must be strictly increasing.");
  AIRT_REQUIRE(o.kmax == K[nK - 1] && o.kmax >= 0, "kmax must equal K(end)");
  AIRT_REQUIRE(o.stoprule == AIRT_STOP_NONE || o.stoprule == AIRT_STOP_DP || o.stoprule == AIRT_STOP_NCP,
               "CART supports the NONE, DP and NCP stopping rules");
  const bool ncp = o.stoprule == AIRT_STOP_NCP;
  if (ncp) {
    AIRT_REQUIRE(o.ncp_rows >= 2 && o.ncp_cols >= 1 && (int64_t)o.ncp_rows * o.ncp_cols == m,
                 "NCP: res_dims must multiply to the number of rows of A");
    AIRT_REQUIRE(o.ncp_smooth >= 1, "NCP: ncp_smooth must be positive");
  }
  AIRT_REQUIRE(o.damp >= 0, "Damping must be positive");
  AIRT_REQUIRE(n < (int64_t)INT32_MAX, "too many columns for CART");
  // the general sweep's shared memory: the block maxima, and the residual too when it fits
  const int64_t nb = (n + kCartBlock - 1) / kCartBlock;
  const size_t smem_r = (size_t)(((nb + 1) & ~(int64_t)1) + std::max<int64_t>(m, 1)) * sizeof(double);
  const bool warp_sweep = smem_r <= kCartSmem;
  const size_t smem = warp_sweep ? smem_r : (size_t)std::max<int64_t>(nb, 1) * sizeof(double);
  AIRT_REQUIRE(smem <= kCartSmem, "CART: too many unknowns for the block maxima in shared memory");
  // always the same limit: other threads may be launching
  AIRT_CHECK_CUDA(cudaFuncSetAttribute(k_cart_sweep_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, kCartSmem));
  AIRT_CHECK_CUDA(cudaFuncSetAttribute(k_cart_sweep_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, kCartSmem));
  const int64_t kmax = o.kmax;

  cudaEvent_t t0, t1;
  AIRT_CHECK_CUDA(cudaEventCreate(&t0));
  AIRT_CHECK_CUDA(cudaEventCreate(&t1));
  AIRT_CHECK_CUDA(cudaEventRecord(t0, s));

  // squared column norms and the column order (cart.m:155-193)
  DevBuf<double> nrm;
  nrm.ensure(std::max<int64_t>(n, 1));
  if (n) {
    k_colnorm2<<<grid_for(n * 32, 256), 256, 0, s>>>(n, P.cp.p, P.cv.p, nrm.p);
    AIRT_LAUNCH_CHECK();
  }
  std::vector<double> hn(n);
  if (n)
    AIRT_CHECK_CUDA(cudaMemcpyAsync(hn.data(), nrm.p, n * sizeof(double), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  std::vector<int> order;
  if (o.order_kind == 0) {
    for (int64_t j = 0; j < n; ++j)
      if (hn[j] > 0) order.push_back((int)j);
  } else {
    AIRT_REQUIRE(o.order_kind == 2 && (o.cols || o.ncols == 0), "column list missing");
    for (int64_t t = 0; t < o.ncols; ++t) {
      const int64_t j = o.cols[t];
      AIRT_REQUIRE(j >= 0 && j < n, "column index out of range");
      if (hn[j] > 0) order.push_back((int)j);
    }
  }
  if (o.damp > 0) {
    double mx = 0;
    for (double v : hn) mx = std::max(mx, v);
    for (double &v : hn) v = v + o.damp * mx;
    nrm.upload(hn.data(), n, s);
  }
  // the blocked sweep needs an order without repeats, (block, row) keys of
  // 32 bits, rows of 27 and a finite relaxpar/||a_j||^2; its inner products
  // take 512 bytes per column
  std::vector<unsigned char> seen(std::max<int64_t>(n, 1), 0);
  bool blocked = !order.empty() && P.nnz < (int64_t)INT32_MAX && m < (int64_t)kCartNoRow &&
                 std::max(bits_for(m), 6) + bits_for((int64_t)(order.size() + kCartCols - 1) / kCartCols) <= 32;
  for (int j : order) {
    blocked = blocked && !seen[j] && std::isfinite(o.relaxpar / hn[j]);
    seen[j] = 1;
  }
  CartPlan &plan = P.cart_plan;
  const bool replan = blocked && !(plan.ready && plan.order == order);
  DevBuf<int> own_cols, nflag, err;
  DevBuf<int> &cols = blocked ? plan.cols : own_cols;
  DevBuf<unsigned char> flag, inorder;
  if (!blocked || replan) {
    if (blocked) plan.ready = false;
    cols.upload(order.data(), order.size(), s);
  }
  nflag.ensure(std::max<int64_t>(n, 1));
  flag.ensure(std::max<int64_t>(n, 1));
  err.ensure(1);
  AIRT_CHECK_CUDA(cudaMemsetAsync(nflag.p, 0, std::max<int64_t>(n, 1) * sizeof(int), s));
  AIRT_CHECK_CUDA(cudaMemsetAsync(flag.p, 1, std::max<int64_t>(n, 1), s));
  AIRT_CHECK_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));

  // x0 and rk = b - A*x0 (cart.m:139)
  P.x64.ensure(std::max<int64_t>(n, 1));
  P.r64.ensure(std::max<int64_t>(m, 1));
  if (d_x0)
    AIRT_CHECK_CUDA(cudaMemcpyAsync(P.x64.p, d_x0, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  else
    AIRT_CHECK_CUDA(cudaMemsetAsync(P.x64.p, 0, std::max<int64_t>(n, 1) * sizeof(double), s));
  if (m) {
    apply_operator(P, P.x64.p, P.r64.p, 0);
    k_sub_from<<<grid_for(m, 256), 256, 0, s>>>(m, d_b, P.r64.p);
    AIRT_LAUNCH_CHECK();
  }
  if (o.lb_kind == AIRT_BOUND_VECTOR) P.lbv.upload(o.lbv, n, s);
  if (o.ub_kind == AIRT_BOUND_VECTOR) P.ubv.upload(o.ubv, n, s);
  DevBuf<double> red;
  red.ensure(1);

  // NCP periodogram of the residual (check_stoprules.m:96-151)
  DevBuf<double> tw, pk, ccol;
  const int q = ncp ? o.ncp_rows / 2 : 0;
  std::vector<double> hcol(ncp ? o.ncp_cols : 0);
  if (ncp) {
    const std::vector<double> tt = ncp_twiddles(o.ncp_rows);
    tw.upload(tt.data(), tt.size(), s);
    pk.ensure((size_t)o.ncp_cols * q);
    ccol.ensure(o.ncp_cols);
  }
  double ncc = 0.0;
  // ||r|| (and the NCP distance) of the residual the sweeps keep
  auto judge_inputs = [&](bool from_sweep) -> double {
    if (!from_sweep) {
      AIRT_CHECK_CUDA(cudaMemsetAsync(red.p, 0, sizeof(double), s));
      if (m) k_sumsq<<<grid_for(m, 256), 256, 0, s>>>(m, P.r64.p, red.p);
      AIRT_LAUNCH_CHECK();
    }
    if (ncp) {
      k_ncp_power<<<dim3(o.ncp_cols, (q + 255) / 256), 256, 0, s>>>(o.ncp_rows, q, P.r64.p, tw.p,
                                                                    pk.p, nullptr);
      k_ncp_col<<<o.ncp_cols, 256, 0, s>>>(q, pk.p, ccol.p, nullptr);
      AIRT_LAUNCH_CHECK();
      AIRT_CHECK_CUDA(cudaMemcpyAsync(hcol.data(), ccol.p, o.ncp_cols * sizeof(double),
                                      cudaMemcpyDeviceToHost, s));
    }
    double h = 0;
    int herr = 0;
    AIRT_CHECK_CUDA(cudaMemcpyAsync(&h, red.p, sizeof(double), cudaMemcpyDeviceToHost, s));
    AIRT_CHECK_CUDA(cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
    AIRT_REQUIRE(!herr, "randi: Nunflag must be a positive integer");
    if (ncp) {
      double sum = 0.0;
      for (double v : hcol) sum += v;
      ncc = sum / o.ncp_cols;
    }
    return std::sqrt(h);
  };

  CartArgs a{};
  a.cp = P.cp.p;
  a.ri = P.ri.p;
  a.cv = P.cv.p;
  a.nrm = nrm.p;
  a.cols = cols.p;
  a.ncols = (int64_t)order.size();
  a.lam = o.relaxpar;
  a.x = P.x64.p;
  a.r = P.r64.p;
  a.flag = flag.p;
  a.nflag = nflag.p;
  a.lbk = o.lb_kind;
  a.ubk = o.ub_kind;
  a.lb = o.lb;
  a.ub = o.ub;
  a.lbv = P.lbv.p;
  a.ubv = P.ubv.p;
  a.thr = o.thr;
  a.kbegin = o.kbegin;
  a.nunflag = o.nunflag;
  a.seed = o.seed;
  a.n = n;
  a.m = m;
  a.r2 = red.p;
  a.err = err.p;

  std::vector<double> resn;
  resn.push_back(judge_inputs(false));
  SweepStop st(o.stoprule, o.taudelta, kmax, o.ncp_smooth);
  st.judge(0, resn[0], ncc);
  CartBlocks B{};
  size_t bsmem = 0;
  const bool rsmem = m <= kCartSharedRows;
  DevBuf<double> od, xold, rold, tail;
  DevBuf<unsigned char> fold;
  DevBuf<int> nfold;
  if (replan && !st.stop) {
    try {
      build_plan(P, a, s);
      plan.order = order;
      plan.ready = true;
    } catch (const Status &e) {
      if (e.code != AIRT_ERR_OOM) throw;
      // no room for the inner products: the general sweep needs none
      plan.cbase.release();
      plan.ent.release();
      plan.gram.release();
      blocked = false;
    }
  }
  if (blocked && !st.stop) {
    od.ensure(order.size());
    B = CartBlocks{plan.nblocks, plan.cbase.p, plan.ent.p, plan.gram.p, od.p};
    bsmem = 4 * kCartCols * kCartCols * sizeof(double) + (rsmem ? (size_t)m * sizeof(double) : 0);
    // always the same limit: other threads may be launching
    AIRT_CHECK_CUDA(cudaFuncSetAttribute(rsmem ? k_cart_block<true> : k_cart_block<false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(4 * kCartCols * kCartCols * sizeof(double) +
                                               kCartSharedRows * sizeof(double))));
    xold.ensure(n);
    rold.ensure(m);
    if (kmax >= o.kbegin) {  // some sweep may flag columns
      fold.ensure(n);
      nfold.ensure(n);
      tail.ensure(order.size());
      inorder.upload(seen.data(), n, s);
    }
  }
  int64_t l = 0;
  auto copy = [&](auto *to, const auto *from, int64_t count) {
    AIRT_CHECK_CUDA(cudaMemcpyAsync(to, from, count * sizeof(*to), cudaMemcpyDeviceToDevice, s));
  };
  for (int64_t k = 1; !st.stop; ++k) {
    // The blocked sweep multiplies inner products with every step of a block,
    // so an infinite or NaN step would reach columns that share no row with
    // it (0 * NaN).  Such a step leaves its trace in the residual: a sweep
    // that starts from or ends with a norm that is not finite is a general one.
    bool finite = blocked && std::isfinite(resn.back());
    double nrk = 0.0;
    if (finite) {
      const bool flags = k >= o.kbegin;  // every flag is set before sweep kbegin
      copy(xold.p, P.x64.p, n);
      copy(rold.p, P.r64.p, m);
      if (flags) {
        copy(fold.p, flag.p, n);
        copy(nfold.p, nflag.p, n);
      }
      if (rsmem) k_cart_block<true><<<1, kCartBlockThreads, bsmem, s>>>(a, B);
      else k_cart_block<false><<<1, kCartBlockThreads, bsmem, s>>>(a, B);
      if (flags) k_cart_flags<<<1, 1024, 0, s>>>(a, k, xold.p, od.p, inorder.p, tail.p);
      AIRT_LAUNCH_CHECK();
      nrk = judge_inputs(true);
      finite = std::isfinite(nrk);
      if (!finite) {
        copy(P.x64.p, xold.p, n);
        copy(P.r64.p, rold.p, m);
        if (flags) {
          copy(flag.p, fold.p, n);
          copy(nflag.p, nfold.p, n);
        }
      }
    }
    if (!finite) {
      if (warp_sweep) k_cart_sweep_warp<<<1, 32, smem, s>>>(a, k);
      else k_cart_sweep_cta<<<1, kCartThreads, smem, s>>>(a, k);
      AIRT_LAUNCH_CHECK();
      nrk = judge_inputs(true);
    }
    resn.push_back(nrk);
    st.judge(k, nrk, ncc);
    if ((l < nK && k == K[l]) || st.stop) {
      AIRT_CHECK_CUDA(cudaMemcpyAsync(d_X + l * n, P.x64.p, n * sizeof(double),
                                      cudaMemcpyDeviceToDevice, s));
      ++l;
    }
  }
  AIRT_CHECK_CUDA(cudaEventRecord(t1, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  float ms = 0;
  cudaEventElapsedTime(&ms, t0, t1);
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  if (resn_host) std::copy(resn.begin(), resn.end(), resn_host);
  if (info) {
    info->stoprule = st.stoprule;
    info->finaliter = st.finaliter;
    info->relaxpar = o.relaxpar;
    info->nsaved = l;
    info->gpu_ms = ms;
  }
}

}  // namespace airt

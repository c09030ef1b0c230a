// Kaczmarz (ART) sweeps on the GPU in the reference's row order
// (art/art.m:227-309).
//
// A sweep is strictly sequential: row step t reads the x that step t-1 wrote.
// Two steps whose rows share no pixel commute exactly, so the order is
// turned into a level schedule: level(t) = 1 + max level of the earlier steps
// that touch one of its pixels.  Steps of one level touch disjoint pixels and
// run concurrently (one warp per step, fixed lane order and shuffle tree, so
// every step computes exactly what it would compute alone); a block barrier
// separates levels.  Each pixel therefore sees the same update sequence, and
// each dot product reads the same values, as in the sequential sweep.
//
// The sweep runs as one launch over all SMs with one warp per step: the steps,
// sorted by level, are dealt round-robin to every warp of the grid, and a step
// waits only until each of its pixels has been written by the earlier steps
// that touch it.  A pixel is a 16-byte word {x, writes so far}, read and
// written by 128-bit accesses, and the schedule holds for every entry how
// many writes must precede it: the poll that finds a pixel ready has its value
// already, and a step publishes its pixels with the stores that write them --
// no completion flags, no fences, no gather after the wait.  The chain of
// levels is the critical path; no grid-wide barrier separates levels.  Each
// wait is bounded: on expiry the kernel raises an error flag, every warp
// leaves, and the host reports AIRT_ERR_TIMEOUT.
//
// Bound: the latency of a level (scattered 128-bit stores, poll, sum), 1.6 us
// with 256 entries per row.  Per sweep, against completion flags per step with
// fences and a gather after the wait: N = 64, 30 angles 0.71 -> 0.30 ms;
// N = 128, 90 angles 1.80 -> 0.74 ms; N = 256, 180 angles 4.58 -> 1.81 ms;
// N = 400, 90 angles (rows past the 512 entries kept in registers) 10.1 -> 7.5.
//
// The whole-vector box projection after every row (art.m:279-284) is
// equivalent to clamping x0 once right after the first row step and the
// row's support after every later step: once x is feasible only the updated
// entries can leave the box.  The first step reads x0 unclamped.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <numeric>

#include "common.cuh"
#include "ncp.cuh"
#include "spmv.cuh"

namespace airt {

namespace {

struct KaczArgs {
  const int64_t *rp;
  const int *ci;
  const float *rv;
  const double *b;
  const double *nrm;
  double lam;
  const double *lam_tab;  // per step of this sweep, or null
  double *x;
  ulonglong2 *xv;         // {x bits, writes in this sweep} of every pixel
  int lbk, ubk;
  double lb, ub;
  const double *lbv, *ubv;
};

__device__ __forceinline__ double clampv(double v, int64_t j, const KaczArgs &a) {
  if (a.lbk == AIRT_BOUND_SCALAR) v = fmax(v, a.lb);
  else if (a.lbk == AIRT_BOUND_VECTOR) v = fmax(v, a.lbv[j]);
  if (a.ubk == AIRT_BOUND_SCALAR) v = fmin(v, a.ub);
  else if (a.ubk == AIRT_BOUND_VECTOR) v = fmin(v, a.ubv[j]);
  return v;
}

// 0: no bounds, 1: scalar bounds only, 2: a vector among them.
__device__ __forceinline__ int clamp_mode(const KaczArgs &a) {
  if (a.lbk == AIRT_BOUND_VECTOR || a.ubk == AIRT_BOUND_VECTOR) return 2;
  return a.lbk != AIRT_BOUND_NONE || a.ubk != AIRT_BOUND_NONE;
}

// Scalar bounds without a branch (a NaN takes the bound, as fmax and fmin do).
__device__ __forceinline__ double clamp_scalar(double v, const KaczArgs &a) {
  v = a.lbk != AIRT_BOUND_NONE && !(v >= a.lb) ? a.lb : v;
  return a.ubk != AIRT_BOUND_NONE && !(v <= a.ub) ? a.ub : v;
}

}  // namespace

// Cycle budget of the bounded waits (the sweep's, and the grid barriers of
// persist.cuh; ~2 s), and a test hook that makes a wait run out: the first
// step waits for a stamp that no step writes, a barrier for an arrival more.
long long g_wait_budget = 4000000000ll;
int g_inject_stall = 0;

namespace {

constexpr int kDagThreads = 256;  // eight warps per CTA

// 128-bit relaxed accesses: one pixel's value and write count together.
struct Pixels {
  ulonglong2 *xv;
  __device__ __forceinline__ ulonglong2 load(int j) const {
    ulonglong2 v;
    asm volatile(
        "{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
        : "=l"(v.x), "=l"(v.y)
        : "l"(xv + j)
        : "memory");
    return v;
  }
  // load_if leaves v alone and store_if does nothing unless `on`; predicated,
  // so that a sequence of them is not cut by branches
  __device__ __forceinline__ void load_if(bool on, int j, ulonglong2 &v) const {
    asm volatile(
        "{ .reg .b128 t; .reg .pred p; setp.ne.s32 p, %3, 0; mov.b128 t, {%0, %1};"
        "  @p ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
        : "+l"(v.x), "+l"(v.y)
        : "l"(xv + j), "r"((int)on)
        : "memory");
  }
  __device__ __forceinline__ void store_if(bool on, int j, double x, unsigned long long writes) const {
    asm volatile(
        "{ .reg .b128 t; .reg .pred p; setp.ne.s32 p, %3, 0; mov.b128 t, {%1, %2};"
        "  @p st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(xv + j),
        "l"(__double_as_longlong(x)), "l"(writes), "r"((int)on)
        : "memory");
  }
};
// Bounded wait of one thread: true while it may go on polling.
struct KaczWait {
  int *err;
  long long budget, t0;
  unsigned n = 0;
  __device__ __forceinline__ bool more() {
    if (++n % 32) return true;
    if (*(volatile int *)err) return false;
    if (clock64() - t0 > budget) {
      atomicExch(err, 1);
      return false;
    }
    return true;
  }
};

struct SweepArgs {
  int nsteps;
  const ArtStep *steps;
  const uint2 *ent;
  int *err;
  long long budget;
  int stall;
};

// One step's operands: the entries of its row (E per lane; longer rows are
// read past them one by one), b, and lambda over the squared norm.
template <int E>
struct KaczRow {
  ArtStep st;
  int cj[E];
  float cv[E];
  unsigned cn[E];
  double bi, lam;
};

__device__ __forceinline__ ArtStep load_step(const SweepArgs &w, int q) {
  ArtStep s{0, 0, 0, 0, 0, -1};
  if (q < w.nsteps) {
    const longlong2 a = __ldg(reinterpret_cast<const longlong2 *>(w.steps + q));
    const int4 b = __ldg(reinterpret_cast<const int4 *>(w.steps + q) + 1);
    s = ArtStep{a.x, a.y, b.x, b.y, b.z, b.w};
  }
  return s;
}

template <int E>
__device__ __forceinline__ void load_row(const SweepArgs &w, const KaczArgs &a, const ArtStep &st, int lane,
                                         KaczRow<E> &r) {
  r.st = st;
#pragma unroll
  for (int u = 0; u < E; ++u) {
    const int e = lane + 32 * u;
    r.cj[u] = 0;
    r.cv[u] = 0.f;
    r.cn[u] = 0;
    if (e < st.len) {
      const uint2 p = __ldg(w.ent + st.off + e);
      r.cj[u] = (int)p.x;
      r.cn[u] = p.y;
      r.cv[u] = __ldg(a.rv + st.s0 + e);
    }
  }
  r.bi = r.lam = 0.0;
  if (st.len) {
    r.bi = __ldg(a.b + st.row);
    // the division leaves the chain of the sweep
    r.lam = (a.lam_tab ? __ldg(a.lam_tab + st.pos) : a.lam) / __ldg(a.nrm + st.row);
  }
}

// Runs one step on the pixels px.  Its loads, sums and stores are free of
// branches: with one per entry they ran one after the other (3.4 ms per sweep
// at N = 256, 180 angles instead of 1.7).  The wait has two parts: a cheap one on the
// entry whose previous writer comes last (rep), until that writer's own
// predecessor is done, and then polls of all entries; with every waiting warp
// polling all of its entries the polls would take bandwidth from the steps
// that run.  Returns false when a wait ran out.
template <int E>
__device__ __forceinline__ bool kacz_step(const SweepArgs &w, const KaczArgs &a, const Pixels &px, KaczRow<E> &r,
                                          int lane, bool stalled, int clamp) {
  const ArtStep &st = r.st;
  const int mine = min(E, (st.len - lane + 31) >> 5);  // entries of this lane
  const unsigned all = mine > 0 ? (1u << mine) - 1u : 0u;
  unsigned waiting = all;
  // the test hook makes the first step wait for a write that never comes
  if (stalled && lane == 0) r.cn[0] += 1;
  KaczWait wait{w.err, w.budget, clock64()};
  bool ok = true;
  if (st.rep >= 0) {
    const uint2 p = __ldg(w.ent + st.off + st.rep);
    while ((unsigned)px.load((int)p.x).y + 1u < p.y && ok) ok = wait.more();
  }
  ulonglong2 v[E];
#pragma unroll
  for (int u = 0; u < E; ++u) v[u] = make_ulonglong2(0ull, 0ull);
  while (ok && waiting) {
#pragma unroll
    for (int u = 0; u < E; ++u) px.load_if(waiting >> u & 1u, r.cj[u], v[u]);
    unsigned ready = 0;
#pragma unroll
    for (int u = 0; u < E; ++u) ready |= ((unsigned)v[u].y == r.cn[u] ? 1u : 0u) << u;
    waiting = all & ~ready;
    if (waiting) ok = wait.more();
  }
  double acc = 0.0, acc1 = 0.0;
#pragma unroll
  for (int u = 0; u < E; u += 2) {  // entries the lane does not have are zero
    acc = fma((double)r.cv[u], __longlong_as_double((long long)v[u].x), acc);
    acc1 = fma((double)r.cv[u + 1], __longlong_as_double((long long)v[u + 1].x), acc1);
  }
  acc += acc1;
  for (int e = lane + 32 * E; ok && e < st.len; e += 32) {
    const uint2 p = __ldg(w.ent + st.off + e);
    ulonglong2 o = px.load((int)p.x);
    while ((unsigned)o.y != p.y && ok) {
      ok = wait.more();
      o = px.load((int)p.x);
    }
    acc = fma((double)__ldg(a.rv + st.s0 + e), __longlong_as_double((long long)o.x), acc);
  }
  if (!__all_sync(0xffffffffu, ok)) return false;
  acc = warp_sum(acc);
  const double c = r.lam * (r.bi - acc);
  double xn[E];
#pragma unroll
  for (int u = 0; u < E; ++u) {
    xn[u] = __dadd_rn(__longlong_as_double((long long)v[u].x), __dmul_rn(c, (double)r.cv[u]));
    if (clamp == 1) xn[u] = clamp_scalar(xn[u], a);
    if (clamp == 2) xn[u] = clampv(xn[u], r.cj[u], a);
  }
#pragma unroll
  for (int u = 0; u < E; ++u) px.store_if(all >> u & 1u, r.cj[u], xn[u], r.cn[u] + 1ull);
  for (int e = lane + 32 * E; e < st.len; e += 32) {
    const int k = (int)__ldg(&w.ent[st.off + e].x);
    const ulonglong2 o = px.load(k);
    double x = __dadd_rn(__longlong_as_double((long long)o.x), __dmul_rn(c, (double)__ldg(a.rv + st.s0 + e)));
    if (clamp) x = clampv(x, k, a);
    px.store_if(true, k, x, o.y + 1ull);
  }
  return true;
}

// One Kaczmarz sweep in the level-sorted step order over all SMs: warp w of the grid (consecutive warps on different SMs)
// runs steps w, w+W, w+2W, ... .
__global__ void __launch_bounds__(kDagThreads, 1) k_kacz_sweep(SweepArgs w, KaczArgs a) {
  const int lane = threadIdx.x & 31;
  const int W = gridDim.x * (blockDim.x >> 5);
  const int clamp = clamp_mode(a);
  for (int q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; q < w.nsteps; q += W) {
    KaczRow<16> r;
    load_row(w, a, load_step(w, q), lane, r);
    if (!kacz_step(w, a, Pixels{a.xv}, r, lane, w.stall && q == 0, clamp)) return;
  }
}

// xv = {x, 0}; and back: x from xv, the write counts zeroed for the next sweep.
__global__ void k_pack_pixels(int n, const double *__restrict__ x, ulonglong2 *__restrict__ xv) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
    xv[j] = make_ulonglong2((unsigned long long)__double_as_longlong(x[j]), 0ull);
}
__global__ void k_unpack_pixels(int n, double *__restrict__ x, ulonglong2 *__restrict__ xv) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    ulonglong2 *p = xv + j;
    x[j] = __longlong_as_double((long long)p->x);
    p->y = 0ull;
  }
}

// Ranks of an order's entries: the pixels in the order of the steps, the start
// of every pixel's run after a stable sort by pixel, and the distance from it.
__global__ void k_order_pixels(int64_t nsteps, const int *__restrict__ order, const int64_t *__restrict__ toff,
                               const int64_t *__restrict__ rp, const int *__restrict__ ci,
                               unsigned *__restrict__ key, unsigned *__restrict__ at) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t t = w; t < nsteps; t += nw) {
    const int64_t s0 = rp[order[t]], len = rp[order[t] + 1] - s0;
    for (int64_t e = lane; e < len; e += 32) {
      key[toff[t] + e] = (unsigned)ci[s0 + e];
      at[toff[t] + e] = (unsigned)(toff[t] + e);
    }
  }
}
__global__ void k_run_starts(int64_t cnt, const unsigned *__restrict__ key, unsigned *__restrict__ start) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < cnt;
       q += (int64_t)gridDim.x * blockDim.x)
    if (q == 0 || key[q] != key[q - 1]) start[key[q]] = (unsigned)q;
}
__global__ void k_ranks(int64_t cnt, const unsigned *__restrict__ key,
                        const unsigned *__restrict__ at, const unsigned *__restrict__ start,
                        uint2 *__restrict__ ent) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < cnt;
       q += (int64_t)gridDim.x * blockDim.x)
    ent[at[q]] = make_uint2(key[q], (unsigned)q - start[key[q]]);
}

// Clamp x0 everywhere except on the support of the first row, whose step
// must read x0 unclamped (one block).
__global__ void __launch_bounds__(1024)
    k_preclamp(int64_t n, int first_row, double *__restrict__ keep, KaczArgs a) {
  const int64_t s0 = a.rp[first_row], s1 = a.rp[first_row + 1];
  for (int64_t e = s0 + threadIdx.x; e < s1; e += blockDim.x) keep[e - s0] = a.x[a.ci[e]];
  __syncthreads();
  for (int64_t j = threadIdx.x; j < n; j += blockDim.x) a.x[j] = clampv(a.x[j], j, a);
  __syncthreads();
  for (int64_t e = s0 + threadIdx.x; e < s1; e += blockDim.x) a.x[a.ci[e]] = keep[e - s0];
}

// ||b - A*x||^2 into *out; with rout the residual itself is kept (NCP).
template <int LANES>
__global__ void __launch_bounds__(256)
    k_resid_norm(int64_t m, const int64_t *__restrict__ rp, const int *__restrict__ ci,
                 const float *__restrict__ rv, const double *__restrict__ x,
                 const double *__restrict__ b, double *__restrict__ out, double *__restrict__ rout) {
  double a = 0;
  for_each_segment<LANES>(m, rp, ci, rv, x, [&](int64_t i, double s, bool lead) {
    if (lead) {
      const double r = b[i] - s;
      a += r * r;
      if (rout) rout[i] = r;
    }
  });
  a = block_sum<256>(a);
  if (threadIdx.x == 0) atomicAdd(out, a);
}

__global__ void k_rownorm2(int64_t m, const int64_t *__restrict__ rp, const float *__restrict__ rv,
                           double *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = w; i < m; i += nw) {
    double a = 0;
    for (int64_t q = rp[i] + lane; q < rp[i + 1]; q += 32) {
      const double v = (double)rv[q];
      a += v * v;
    }
    a = warp_sum(a);
    if (lane == 0) out[i] = a;
  }
}

__global__ void k_copy_d(int64_t n, const double *__restrict__ a, double *__restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    b[i] = a[i];
}

using Schedule = ArtSchedule;

// Ranks of an order's entries on the device: two sorts' worth of work space,
// 24-32 bytes per entry, for fewer than 2^32 entries.
void rank_entries(Problem &P, const std::vector<int> &ord, const std::vector<int64_t> &toff, int64_t cnt, int64_t n,
                  Schedule &S, cudaStream_t s) {
  const int64_t nsteps = (int64_t)ord.size();
  DevBuf<int> dord;
  DevBuf<int64_t> dtoff;
  DevBuf<unsigned> key, key2, at, at2, start;
  DevBuf<unsigned char> tmp;
  dord.upload(ord.data(), nsteps, s);
  dtoff.upload(toff.data(), nsteps + 1, s);
  key.ensure(cnt);
  key2.ensure(cnt);
  at.ensure(cnt);
  at2.ensure(cnt);
  start.ensure(n);
  k_order_pixels<<<grid_for(nsteps * 32, 256), 256, 0, s>>>(nsteps, dord.p, dtoff.p, P.rp.p, P.ci.p, key.p, at.p);
  AIRT_LAUNCH_CHECK();
  int bits = 1;
  while (bits < 31 && (1ll << bits) < n) ++bits;
  size_t need = 0;
  AIRT_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, need, key.p, key2.p, at.p, at2.p, cnt, 0, bits, s));
  tmp.ensure(need);
  AIRT_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, need, key.p, key2.p, at.p, at2.p, cnt, 0, bits, s));
  const unsigned g = grid_for(cnt, 256);
  k_run_starts<<<g, 256, 0, s>>>(cnt, key2.p, start.p);
  k_ranks<<<g, 256, 0, s>>>(cnt, key2.p, at2.p, start.p, S.ent.p);
  AIRT_LAUNCH_CHECK();
}

// The same on the host, where the device has no room for the sort or the
// order visits more entries than it numbers; copied in slices.
void rank_on_host(const std::vector<int64_t> &hrp, const std::vector<int> &hci, const std::vector<int> &ord,
                  int64_t n, Schedule &S, cudaStream_t s) {
  constexpr size_t kSlice = 4 << 20;
  std::vector<unsigned> writes(n, 0);
  std::vector<uint2> buf;
  int64_t done = 0;
  auto flush = [&] {
    AIRT_CHECK_CUDA(cudaMemcpyAsync(S.ent.p + done, buf.data(), buf.size() * sizeof(uint2), cudaMemcpyHostToDevice, s));
    AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
    done += (int64_t)buf.size();
    buf.clear();
  };
  for (const int row : ord)
    for (int64_t e = hrp[row]; e < hrp[row + 1]; ++e) {
      buf.push_back(make_uint2((unsigned)hci[e], writes[hci[e]]++));
      if (buf.size() == kSlice) flush();
    }
  flush();
}

// Level schedule of a row order (see the file comment): the levels on the
// host, the entries' ranks on the device.
void build_schedule(Problem &P, const std::vector<int64_t> &hrp, const std::vector<int> &hci,
                    const int64_t *order, int64_t nsteps, int64_t n, Schedule &S, cudaStream_t s) {
  std::vector<int> level(nsteps), last(n, -1), rept(nsteps), ord(nsteps);
  std::vector<int64_t> toff(nsteps + 1, 0);
  int maxlev = -1;
  for (int64_t t = 0; t < nsteps; ++t) {
    const int64_t row = order[t], e0 = hrp[row], e1 = hrp[row + 1];
    int L = -1, at = -1;  // highest level that wrote one of the row's pixels
    for (int64_t e = e0; e < e1; ++e) {
      const int v = last[hci[e]];
      if (v > L) {
        L = v;
        at = (int)(e - e0);
      }
    }
    ++L;
    for (int64_t e = e0; e < e1; ++e) last[hci[e]] = L;
    level[t] = L;
    rept[t] = at;
    ord[t] = (int)row;
    toff[t + 1] = toff[t] + (e1 - e0);
    maxlev = std::max(maxlev, L);
  }
  S.nlev = maxlev + 1;
  S.nsteps = nsteps;
  const int64_t cnt = toff[nsteps];
  std::vector<int> ptr(S.nlev + 1, 0);
  std::vector<ArtStep> steps(nsteps);
  for (int64_t t = 0; t < nsteps; ++t) ++ptr[level[t] + 1];
  for (int L = 0; L < S.nlev; ++L) ptr[L + 1] += ptr[L];
  for (int64_t t = 0; t < nsteps; ++t) {
    const int64_t row = order[t];
    steps[ptr[level[t]]++] =
        ArtStep{hrp[row], toff[t], (int)(hrp[row + 1] - hrp[row]), (int)row, (int)t, rept[t]};
  }
  S.steps.upload(steps.data(), nsteps, s);
  S.ent.ensure(cnt);
  bool ranked = cnt == 0;
  if (!ranked && cnt < (int64_t)UINT32_MAX) {
    try {
      rank_entries(P, ord, toff, cnt, n, S, s);
      ranked = true;
    } catch (const Status &e) {
      if (e.code != AIRT_ERR_OOM) throw;
    }
  }
  if (!ranked) rank_on_host(hrp, hci, ord, n, S, s);
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));  // the host vectors and work space end here
}

}  // namespace

void run_art(Problem &P, const airt_art_opts &o, const double *d_b, const double *d_x0,
             const int64_t *K, int64_t nK, double *d_X, double *resn_host, airt_info *info) {
  cudaStream_t s = P.stream;
  const int64_t m = P.m, n = P.n;
  AIRT_REQUIRE(!P.matrix_free, "ART needs the stored matrix (row access)");
  AIRT_REQUIRE(nK >= 1 && K, "Max no. of iterations must ALWAYS be specified.");
  for (int64_t l = 1; l < nK; ++l)
    AIRT_REQUIRE(K[l] > K[l - 1], "Elements of K must be strictly increasing.");
  AIRT_REQUIRE(o.kmax == K[nK - 1] && o.kmax >= 0, "kmax must equal K(end)");
  AIRT_REQUIRE(o.stoprule == AIRT_STOP_NONE || o.stoprule == AIRT_STOP_DP || o.stoprule == AIRT_STOP_NCP,
               "ART supports the NONE, DP and NCP stopping rules");
  const bool ncp = o.stoprule == AIRT_STOP_NCP;
  if (ncp) {
    AIRT_REQUIRE(o.ncp_rows >= 2 && o.ncp_cols >= 1 && (int64_t)o.ncp_rows * o.ncp_cols == m,
                 "NCP: res_dims must multiply to the number of rows of A");
    AIRT_REQUIRE(o.ncp_smooth >= 1, "NCP: ncp_smooth must be positive");
  }
  AIRT_REQUIRE(o.damp >= 0, "Damping must be positive");
  AIRT_REQUIRE(m < (int64_t)INT32_MAX, "too many rows for ART");
  const int64_t kmax = o.kmax;

  cudaEvent_t t0, t1;
  AIRT_CHECK_CUDA(cudaEventCreate(&t0));
  AIRT_CHECK_CUDA(cudaEventCreate(&t1));
  AIRT_CHECK_CUDA(cudaEventRecord(t0, s));

  // squared row norms (art.m:161-181) and damping (art.m:206)
  DevBuf<double> nrm;
  nrm.ensure(m);
  k_rownorm2<<<grid_for(m * 32, 256), 256, 0, s>>>(m, P.rp.p, P.rv.p, nrm.p);
  AIRT_LAUNCH_CHECK();
  std::vector<double> hn(m);
  AIRT_CHECK_CUDA(cudaMemcpyAsync(hn.data(), nrm.p, m * sizeof(double), cudaMemcpyDeviceToHost, s));
  AIRT_CHECK_CUDA(cudaStreamSynchronize(s));

  // row order (art.m:183-203)
  std::vector<int64_t> I;
  for (int64_t i = 0; i < m; ++i)
    if (hn[i] > 0) I.push_back(i);
  std::vector<int64_t> order;
  int64_t stride = 0;
  if (o.order_kind == 0) {
    order = I;
  } else if (o.order_kind == 1) {
    order = I;
    order.insert(order.end(), I.rbegin(), I.rend());
  } else {
    AIRT_REQUIRE(o.rows && o.nrows >= 0, "row list missing");
    stride = o.rows_stride;
    const int64_t lists = stride > 0 ? kmax : 1;
    for (int64_t k = 0; k < lists; ++k) {
      for (int64_t t = 0; t < o.nrows; ++t) {
        const int64_t r = o.rows[k * stride + t];
        AIRT_REQUIRE(r >= 0 && r < m, "row index out of range");
        if (hn[r] > 0) order.push_back(r);
      }
    }
  }
  if (o.damp > 0) {
    double mx = 0;
    for (double v : hn) mx = std::max(mx, v);
    for (double &v : hn) v = v + o.damp * mx;
    nrm.upload(hn.data(), m, s);
  }
  const int64_t per_sweep =
      (o.order_kind == 2 && stride > 0) ? (int64_t)order.size() / std::max<int64_t>(kmax, 1)
                                        : (int64_t)order.size();
  AIRT_REQUIRE(o.order_kind != 2 || stride == 0 || (int64_t)order.size() == per_sweep * kmax,
               "each sweep of the row stream must keep the same number of nonzero rows");

  // the schedule of a fixed order is kept in the problem and rebuilt only for
  // a new order; per-sweep orders (a row stream) get one per sweep
  const bool per_sweep_sched = (o.order_kind == 2 && stride > 0);
  Schedule local;
  Schedule &S = per_sweep_sched ? local : P.art_sched;
  const bool need_pattern = per_sweep_sched || !S.ready || (int64_t)S.order.size() != per_sweep ||
                            !std::equal(S.order.begin(), S.order.end(), order.begin());
  // host copy of the sparsity pattern, only when a schedule is built
  std::vector<int64_t> hrp;
  std::vector<int> hci;
  if (need_pattern) {
    hrp.resize(m + 1);
    hci.resize(P.nnz);
    AIRT_CHECK_CUDA(cudaMemcpyAsync(hrp.data(), P.rp.p, (m + 1) * sizeof(int64_t),
                                    cudaMemcpyDeviceToHost, s));
    if (P.nnz)
      AIRT_CHECK_CUDA(cudaMemcpyAsync(hci.data(), P.ci.p, P.nnz * sizeof(int), cudaMemcpyDeviceToHost, s));
    AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
  }
  if (!per_sweep_sched && need_pattern) {
    S.ready = false;
    build_schedule(P, hrp, hci, order.data(), per_sweep, n, S, s);
    S.order.assign(order.begin(), order.begin() + per_sweep);
    S.ready = true;
  }

  // iterate
  P.x64.ensure(n);
  if (d_x0)
    k_copy_d<<<grid_for(n, 256), 256, 0, s>>>(n, d_x0, P.x64.p);
  else
    AIRT_CHECK_CUDA(cudaMemsetAsync(P.x64.p, 0, n * sizeof(double), s));
  if (o.lb_kind == AIRT_BOUND_VECTOR) P.lbv.upload(o.lbv, n, s);
  if (o.ub_kind == AIRT_BOUND_VECTOR) P.ubv.upload(o.ubv, n, s);
  // sweep kernel: pixels with their write counts, error flag, grid size
  DevBuf<ulonglong2> xv;
  xv.ensure(std::max<int64_t>(n, 1));
  P.err.ensure(1);
  AIRT_CHECK_CUDA(cudaMemsetAsync(P.err.p, 0, sizeof(int), s));
  int occ = 0;
  AIRT_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_kacz_sweep, kDagThreads, 0));
  AIRT_REQUIRE(occ >= 1, "the Kaczmarz sweep kernel cannot be resident");
  const int dag_grid = num_sms();
  const long long budget = g_wait_budget;
  const int stall = g_inject_stall;
  int herr = 0;
  DevBuf<double> tab, red, keep;
  if (o.relax_table && kmax > 0) tab.upload(o.relax_table, kmax * per_sweep, s);
  red.ensure(1);
  keep.ensure(std::max<int64_t>(P.N ? 2 * P.N + 2 : 1, 1));

  KaczArgs a{};
  a.rp = P.rp.p;
  a.ci = P.ci.p;
  a.rv = P.rv.p;
  a.b = d_b;
  a.nrm = nrm.p;
  a.lam = o.relaxpar;
  a.x = P.x64.p;
  a.xv = xv.p;
  a.lbk = o.lb_kind;
  a.ubk = o.ub_kind;
  a.lb = o.lb;
  a.ub = o.ub;
  a.lbv = P.lbv.p;
  a.ubv = P.ubv.p;

  const int L = lanes_for(P.nnz, m);
  // NCP: the residual, the periodogram distances per column, and the
  // ncp_smooth history (check_inputs.m:209, +inf initially)
  DevBuf<double> r64, tw, pk, ccol;
  const int q = ncp ? o.ncp_rows / 2 : 0;
  std::vector<double> hcol(ncp ? o.ncp_cols : 0);
  if (ncp) {
    r64.ensure(m);
    const std::vector<double> t = ncp_twiddles(o.ncp_rows);
    tw.upload(t.data(), t.size(), s);
    pk.ensure((size_t)o.ncp_cols * q);
    ccol.ensure(o.ncp_cols);
  }
  double ncc = 0.0;
  auto resid = [&]() -> double {
    AIRT_CHECK_CUDA(cudaMemsetAsync(red.p, 0, sizeof(double), s));
    const unsigned g = grid_for(m * L, 256);
    switch (L) {
      case 32: k_resid_norm<32><<<g, 256, 0, s>>>(m, P.rp.p, P.ci.p, P.rv.p, P.x64.p, d_b, red.p, ncp ? r64.p : nullptr); break;
      case 16: k_resid_norm<16><<<g, 256, 0, s>>>(m, P.rp.p, P.ci.p, P.rv.p, P.x64.p, d_b, red.p, ncp ? r64.p : nullptr); break;
      case 8: k_resid_norm<8><<<g, 256, 0, s>>>(m, P.rp.p, P.ci.p, P.rv.p, P.x64.p, d_b, red.p, ncp ? r64.p : nullptr); break;
      default: k_resid_norm<4><<<g, 256, 0, s>>>(m, P.rp.p, P.ci.p, P.rv.p, P.x64.p, d_b, red.p, ncp ? r64.p : nullptr); break;
    }
    AIRT_LAUNCH_CHECK();
    if (ncp) {
      k_ncp_power<<<dim3(o.ncp_cols, (q + 255) / 256), 256, 0, s>>>(o.ncp_rows, q, r64.p, tw.p, pk.p, nullptr);
      k_ncp_col<<<o.ncp_cols, 256, 0, s>>>(q, pk.p, ccol.p, nullptr);
      AIRT_LAUNCH_CHECK();
      AIRT_CHECK_CUDA(cudaMemcpyAsync(hcol.data(), ccol.p, o.ncp_cols * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    double h = 0;
    AIRT_CHECK_CUDA(cudaMemcpyAsync(&h, red.p, sizeof(double), cudaMemcpyDeviceToHost, s));
    AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
    if (ncp) {
      double sum = 0.0;
      for (double v : hcol) sum += v;
      ncc = sum / o.ncp_cols;
    }
    return std::sqrt(h);
  };

  std::vector<double> resn;
  resn.push_back(resid());
  SweepStop st(o.stoprule, o.taudelta, kmax, o.ncp_smooth);
  st.judge(0, resn[0], ncc);
  int64_t l = 0;
  const bool bounded = o.lb_kind != AIRT_BOUND_NONE || o.ub_kind != AIRT_BOUND_NONE;
  double lam_last = o.relaxpar;
  for (int64_t k = 1; !st.stop; ++k) {
    const int64_t *ord = order.data() + (per_sweep_sched ? (k - 1) * per_sweep : 0);
    if (per_sweep_sched) build_schedule(P, hrp, hci, ord, per_sweep, n, S, s);
    if (k == 1 && bounded && per_sweep > 0) {
      const int64_t r0 = ord[0];
      int64_t rr[2];
      AIRT_CHECK_CUDA(cudaMemcpyAsync(rr, P.rp.p + r0, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
      AIRT_CHECK_CUDA(cudaStreamSynchronize(s));
      const int64_t len = rr[1] - rr[0];
      keep.ensure(std::max<int64_t>(len, 1));
      k_preclamp<<<1, 1024, 0, s>>>(n, (int)r0, keep.p, a);
    }
    a.lam_tab = tab.p ? tab.p + (k - 1) * per_sweep : nullptr;
    if (S.nsteps > 0) {
      const SweepArgs w{(int)S.nsteps, S.steps.p, S.ent.p, P.err.p, budget, stall};
      if (k == 1) k_pack_pixels<<<grid_for(n, 256), 256, 0, s>>>((int)n, P.x64.p, xv.p);
      void *args[] = {(void *)&w, &a};
      AIRT_CHECK_CUDA(cudaLaunchCooperativeKernel((const void *)k_kacz_sweep, dim3(dag_grid),
                                                  dim3(kDagThreads), args, 0, s));
      k_unpack_pixels<<<grid_for(n, 256), 256, 0, s>>>((int)n, P.x64.p, xv.p);
    }
    AIRT_LAUNCH_CHECK();
    AIRT_CHECK_CUDA(cudaMemcpyAsync(&herr, P.err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    if (o.relax_table && per_sweep > 0) lam_last = o.relax_table[(k - 1) * per_sweep + per_sweep - 1];
    const double nrk = resid();  // synchronises the stream (herr is current)
    if (herr) {
      cudaEventDestroy(t0);
      cudaEventDestroy(t1);
      set_error("a bounded device wait of the Kaczmarz sweep gave up (sweep %lld)", (long long)k);
      throw Status{AIRT_ERR_TIMEOUT};
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
    info->relaxpar = lam_last;
    info->nsaved = l;
    info->gpu_ms = ms;
  }
}

}  // namespace airt

extern "C" int airt_test_set_wait_budget(long long cycles) {
  if (cycles <= 0) return AIRT_ERR_ARG;
  airt::g_wait_budget = cycles;
  return AIRT_OK;
}

extern "C" int airt_test_inject_stall(int on) {
  airt::g_inject_stall = on ? 1 : 0;
  return AIRT_OK;
}

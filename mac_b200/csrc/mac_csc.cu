// The drop-in linear solver's Jacobi-PCG as one resident kernel per solve.
//
// The pressure matrices the reference hands over have thousands to a few
// hundred thousand rows of at most seven entries, so an iteration moves a few
// megabytes at most and its time is the latency of launches, reductions and
// host reads: four launches, a memset and two host reads of the scalars took
// 60 us an iteration whatever the size. Here a row stays with one thread for
// the whole solve (its entries, its x, r, p and its copies of the neighbours' p,
// in registers but for what the compiler spills: 128 bytes stored and 80 loaded in
// the code of the form with 128 registers, 356 and 256 in that with 64), the blocks of
// one cooperative launch exchange the two dot products of an iteration through
// tagged slots, and only z = D^-1 r passes through memory (L2), as tagged words
// like the dots: no fence, no barrier. Measured on one B200, factorise and solve,
// launches and this kernel: n = 40,960 (127 iterations) 8.1 and 1.2 ms; with two
// blocks an SM 79,507 (132) 9.4 and 2.2 ms, 148,877 (143) 11.4 and 3.4 ms.
#include <cmath>

#include "mac_internal.cuh"

namespace mac {

constexpr int kCgThreads = 512;
constexpr int kCgRow = kCscRow;      // entries of a row held in registers (the 7-point stencil)
constexpr int kCgMaxBlocks = 512;    // blocks whose slots one block's threads can poll
constexpr int kCgSpin = kWaitPolls;  // polls before a wait for the other blocks gives up
// Each block's slot has a 128-byte line to itself: with 32-byte slots the
// polls of one line by all blocks queued behind each other (an exchange among
// 148 blocks took 2.4 us, against 1.0 us with a line each).
constexpr int kCgSlot = 16;

// A double in two 64-bit words that each carry half of it and a tag: a reader
// polls the data itself until both tags match, so publishing a value needs no
// fence and no flag (each word is read and written whole).
__device__ __forceinline__ void ll_store(unsigned long long* s, double v, unsigned tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(s), "l"(t | (b >> 32)),
               "l"(t | (b & 0xffffffffull))
               : "memory");
}
__device__ __forceinline__ bool ll_load(const unsigned long long* s, unsigned tag, double* v) {
  unsigned long long a, b;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(s) : "memory");
  *v = __longlong_as_double((long long)((a << 32) | (b & 0xffffffffull)));
  return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}

// Sums a (and b when TWO) over the whole grid, in block order, the same value
// in every thread. Slots alternate between two sets: a block posts exchange t
// only after it has read every block's t - 1, and each of those was posted
// after its block had read t - 2. One warp posts and polls while the others
// wait at a barrier: warps left to run on into the next phase queued their
// loads before the polls (7.6 us an iteration at 97 blocks instead of 5.0).
// False when the bounded wait ran out.
template <bool TWO>
__device__ inline bool grid_sum(double& a, double& b, unsigned long long* slots, unsigned tag) {
  constexpr int W = kCgThreads / 32, U = 4;  // U slots a lane in flight
  __shared__ double sa[W], sb[W], tot[2];
  __shared__ int sok;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, s);
    if (TWO) b += __shfl_down_sync(0xffffffffu, b, s);
  }
  if (lane == 0) {
    sa[w] = a;
    if (TWO) sb[w] = b;
  }
  __syncthreads();
  if (w == 0) {
    unsigned long long* set = slots + (size_t)(tag & 1) * kCgSlot * G;
    a = lane < W ? sa[lane] : 0.0;
    if (TWO) b = lane < W ? sb[lane] : 0.0;
#pragma unroll
    for (int s = W / 2; s > 0; s >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, s);
      if (TWO) b += __shfl_down_sync(0xffffffffu, b, s);
    }
    if (lane == 0) {
      ll_store(set + kCgSlot * blockIdx.x, a, tag);
      if (TWO) ll_store(set + kCgSlot * blockIdx.x + 2, b, tag);
    }
    a = 0;
    b = 0;
    bool ok = true;
    for (int g0 = 0; g0 < G && ok; g0 += 32 * U) {
      double va[U], vb[U];
      ok = false;
      for (int i = 0; i < kCgSpin && !ok; ++i) {
        ok = true;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int g = g0 + 32 * u + lane;
          va[u] = vb[u] = 0;
          if (g >= G) continue;
          ok = ll_load(set + kCgSlot * g, tag, &va[u]) && ok;
          if (TWO) ok = ll_load(set + kCgSlot * g + 2, tag, &vb[u]) && ok;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        a += va[u];
        if (TWO) b += vb[u];
      }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, s);
      if (TWO) b += __shfl_down_sync(0xffffffffu, b, s);
    }
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) {
      tot[0] = a;
      tot[1] = b;
      sok = ok;
    }
  }
  __syncthreads();
  a = tot[0];
  if (TWO) b = tot[1];
  return sok != 0;
}

// Row j = blockIdx 512 + threadIdx. out: iterations, r.r, b.b and 1 when a
// wait ran out. flags[0] != 0 (the matrix is not of the form CG needs) or
// flags[1] != 0 (a row of more than kCgRow entries): nothing is done. z holds
// two tagged words a row: a row's z of an iteration is overwritten only after
// the next p.q exchange, which every block enters with its neighbours' z read.
// Two blocks an SM (64 registers) where the rows need them, else one.
template <int MINB>
__global__ void __launch_bounds__(kCgThreads, MINB) k_csc_cg(int n, const int* __restrict__ off,
                                                             const int* __restrict__ ind,
                                                             const double* __restrict__ val,
                                                             const double* __restrict__ bv, double* x,
                                                             unsigned long long* z, unsigned long long* slots,
                                                             const double* flags, double rtol2, int max_iters,
                                                             int polls, double* out) {
  if (flags && (flags[0] != 0.0 || flags[1] != 0.0)) return;
  __shared__ int late;  // a thread of the block gave up waiting for a neighbour's z
  if (threadIdx.x == 0) late = 0;
  const int j = blockIdx.x * kCgThreads + threadIdx.x;
  const bool live = j < n;
  int nb[kCgRow];
  double av[kCgRow], pn[kCgRow], dinv = 0, r = 0, p = 0, xs = 0, s0 = 0, s1 = 0;
  const int k0 = live ? off[j] : 0, len = live ? off[j + 1] - k0 : 0;
#pragma unroll
  for (int m = 0; m < kCgRow; ++m) {
    nb[m] = m < len ? ind[k0 + m] : -1;
    av[m] = m < len ? val[k0 + m] : 0.0;
    pn[m] = 0;
    if (nb[m] == j) dinv = -av[m];
  }
  unsigned tag = 1;
  if (live) {
    dinv = dinv != 0 ? 1.0 / dinv : 0.0;
    const double b0 = bv[j];
    r = -b0;
    p = dinv * r;
    ll_store(z + 2 * (size_t)j, p, tag);
    s0 = r * p;
    s1 = b0 * b0;
  }
  bool ok = grid_sum<true>(s0, s1, slots, tag);
  double rz = s0, rr = s1, beta = 0;
  const double bb = s1;
  int it = 0;
  while (ok && bb > 0 && it < max_iters) {
    // the neighbours' p = z + beta p, formed here as their own row forms it
    double q = 0;
    bool got = false;
    for (int i = 0; i < polls && !got; ++i) {
      double zn[kCgRow];
      got = true;
#pragma unroll
      for (int m = 0; m < kCgRow; ++m)
        if (nb[m] >= 0) got = ll_load(z + 2 * (size_t)nb[m], tag, &zn[m]) && got;
      if (!got) continue;
#pragma unroll
      for (int m = 0; m < kCgRow; ++m)
        if (nb[m] >= 0) {
          pn[m] = zn[m] + beta * pn[m];
          q += av[m] * pn[m];
        }
    }
    // M = -A; the NaN of a wait that ran out ends every block's solve
    q = got ? -q : __longlong_as_double(0x7ff8000000000000ll);
    s0 = p * q;
    ok = grid_sum<false>(s0, s1, slots, ++tag);
    // breakdown: x keeps the last finite iterate. Whether it was a wait is asked here
    // only: as part of every iteration's test it took 4% of one
    if (!ok || !(s0 != 0.0 && isfinite(s0))) {
      if (!got) late = 1;
      __syncthreads();
      break;
    }
    const double alpha = rz / s0;
    xs += alpha * p;
    r -= alpha * q;
    const double zk = dinv * r;
    ++tag;
    if (live) ll_store(z + 2 * (size_t)j, zk, tag);
    s0 = r * zk;
    s1 = r * r;
    ok = grid_sum<true>(s0, s1, slots, tag);
    if (!ok) break;
    ++it;
    rr = s1;
    if (rr <= rtol2 * bb) break;
    beta = s0 / rz;
    rz = s0;
    p = zk + beta * p;
  }
  if (live) x[j] = xs;
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    out[0] = it;
    out[1] = rr;
    out[2] = bb;
  }
  if (threadIdx.x == 0 && (!ok || late)) out[3] = 1.0;
}

// Enqueues the whole solve of A x = b (A symmetric with a negative diagonal,
// rows of at most kCgRow entries) on st: `work` (16-byte aligned) holds 2 n
// doubles of tagged z and kCscWork more, res (4 doubles) receives iterations,
// r.r, b.b and a timeout mark; polls bounds the wait for a neighbour's z.
// *enqueued = 0 when the driver refuses the launch or the system does not fit the
// resident form: a row a thread and two blocks an SM hold 151,552 rows on 148
// SMs, and a block polls at most kCgMaxBlocks slots.
int csc_cg_resident(cudaStream_t st, int n, const int* off, const int* ind, const double* val, const double* b,
                    double* x, double* work, const double* flags, double rtol, int max_iters, int polls,
                    double* res, int* enqueued) {
  *enqueued = 0;
  int dev = 0, nsm = 0, occ = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) || !coop ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_csc_cg<2>, kCgThreads, 0))
    return MAC_OK;
  const int g = (n + kCgThreads - 1) / kCgThreads;
  if (g > nsm * occ || g > kCgMaxBlocks) return MAC_OK;
  unsigned long long *z = reinterpret_cast<unsigned long long*>(work), *slots = z + 2 * (size_t)n;
  int rc = check(cudaMemsetAsync(z, 0, 16 * (size_t)n + 2 * 8 * kCgSlot * (size_t)g, st));  // no tag is 0
  if (!rc) rc = check(cudaMemsetAsync(res, 0, 32, st));
  if (rc) return rc;
  double rtol2 = rtol * rtol;
  void* args[] = {&n, &off, &ind, &val, &b, &x, &z, &slots, &flags, &rtol2, &max_iters, &polls, &res};
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.gridDim = g;
  cfg.blockDim = kCgThreads;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  launch_resident(cfg, g <= nsm ? (const void*)k_csc_cg<1> : (const void*)k_csc_cg<2>, args, enqueued);
  return MAC_OK;
}

// flags (zeroed before): [0] the matrix is not symmetric with exactly one
// negative diagonal entry a column (or its arrays are not valid), [1] a column
// of more than kCgRow entries, [2] (REPEATS only) a column repeats a row, so that
// the entry by entry comparison decides nothing. Column i is scanned linearly for the
// mirror entry (the reference's columns hold at most 7). The search for repeats
// takes the square of a column's length, so only the caller that acts on it
// asks for it, for valid arrays and columns whose length it has bounded.
template <bool REPEATS>
__global__ void k_csc_check(int n, const int* __restrict__ off, const int* __restrict__ ind,
                            const double* __restrict__ val, double* flags) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int k0 = off[j], k1 = off[j + 1];
    bool bad = j == 0 && k0 != 0;
    int ndiag = 0;
    if (k1 < k0) bad = true;
    if (k1 - k0 > kCgRow) flags[1] = 1.0;
    for (int k = k0; k < k1 && !bad; ++k) {
      const int i = ind[k];
      if (i < 0 || i >= n) {
        bad = true;
      } else if (i == j) {
        ndiag += 1;
        if (!(val[k] < 0)) bad = true;
      } else {
        bool found = false;
        for (int m = off[i]; m < off[i + 1]; ++m)
          if (ind[m] == j) {
            found = val[m] == val[k];
            break;
          }
        if (!found) bad = true;
      }
    }
    // all pairs of the column, whatever the comparison met: a coupling in unequal
    // parts differs from its mirror's first part and is equal all the same
    if (REPEATS)
      for (int k = k0 + 1; k < k1; ++k)
        for (int m = k0; m < k; ++m)
          if (ind[m] == ind[k]) flags[2] = 1.0;
    if (bad || ndiag != 1) flags[0] = 1.0;
  }
}
template __global__ void k_csc_check<false>(int, const int*, const int*, const double*, double*);
template __global__ void k_csc_check<true>(int, const int*, const int*, const double*, double*);

}  // namespace mac

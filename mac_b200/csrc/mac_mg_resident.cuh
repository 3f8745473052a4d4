// The whole MG-PCG solve as one resident kernel, for systems of up to about a
// thousand bricks. Included by mac_mg.cu.
//
// A CG iteration of the launch-by-launch form is some twenty dependent kernels,
// each a few microseconds of launch, ramp-up and one or two rounds of load
// latency, so an iteration took 65-80 us however small the system was. Here one
// block an SM (or one cluster of up to 16 blocks, for the smallest systems) runs
// every phase of every iteration; phases are separated by a grid-wide exchange
// that also carries the dot products, static data of the next phase is loaded
// while a block waits, the coarse levels stay in block 0's shared memory for the
// whole solve, and the host reads the scalars once, at the end. What bounds an
// iteration now is the latency of its 10 (level 2 in block 0) or 14 exchanges
// and of the one or two rounds of L2 loads behind each. Measured a CG iteration
// on one B200, before and after: 3,439 unknowns (FP32 levels) 65 -> 23 us, 9,042
// (FP64) 70 -> 25, 52,857 (FP64) 75 -> 36, 315,783 (FP32) 77 -> 52.
//
// The arithmetic of a phase is that of the kernel it stands for (k0_pre,
// k0_restrict, kl_*, k0_post, k_update_spmv), cell for cell; the dot products
// add in block order, which depends on the system's size alone.

constexpr int kResThreads = 512;                 // 128 registers a thread (spills are reloaded from L2 after every exchange)
constexpr int kResGroups = kResThreads / 128;    // bricks a block works on at once
constexpr int kResWarps = kResThreads / 32;
constexpr int kResCluster = 16;                  // blocks of the one-cluster form

template <class T>
struct ResArgs {
  const int* drow;
  int nd;
  const uint16_t* fmask;
  double *r, *r2, *x, *pd, *pd2, *q, *z;
  T *e0, *e0b, *e1, *e1b, *e2, *e2b, *r1, *r2l;
  const T *w1, *w2;
  size_t ncap1, ncap2;
  DenseSet<T> S;     // dense levels (level 3 and below), solved by block 0 in shared memory
  int l2;            // 1: so is level 2, as a dense grid of 2 x 2 x 2 cells a brick of the box
  const double* inv;
  const int* inv_ok;
  Scalars* ds;
  unsigned long long* slots;
  Params P;
  double rtol2;
  int max_iters;
  int polls;         // after which a wait for the other blocks gives up
  size_t blk_bytes;  // shared memory of block 0's levels
  int cluster;       // 1: launched as one cluster
};

// ---- exchange: a grid barrier that can sum one double over the blocks
// Blocks of the whole grid count arrivals in one word (release) and one thread
// a block polls it (acquire); a sum's parts go to slots read after the wait.
// Against tagged slots polled by a warp, which need a fence on either side to
// publish the phase's data, a phase takes 1.9 instead of 2.9 us at 148 blocks.
// In one cluster the hardware barrier does both (0.25 us) and the parts go
// through distributed shared memory.
struct ResSync {
  unsigned* counter;   // arrivals since the context was made
  double* parts;       // [2][gridDim] parts of the last two sums
  unsigned target;
  unsigned parity;
  int cluster;
  int polls;
  double* red;         // [kResWarps] warp sums, then [2][kResCluster] the cluster's slots (grid: the total)
  int* ok;
};

// Everything the block wrote is published with its part of the sum; what the
// block loads between res_arrive and res_wait must be static.
template <bool SUM>
__device__ __forceinline__ void res_arrive(ResSync& y, double v) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  y.target += gridDim.x;
  y.parity ^= 1;
  if (SUM) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
    if (lane == 0) y.red[w] = v;
  }
  if (SUM || !y.cluster) __syncthreads();
  if (w == 0) {
    if (SUM) {
      v = lane < kResWarps ? y.red[lane] : 0.0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
      v = __shfl_sync(0xffffffffu, v, 0);
    }
    if (!y.cluster) {
      if (lane == 0) {
        if (SUM) y.parts[y.parity * gridDim.x + blockIdx.x] = v;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(y.counter) : "memory");
      }
    } else if (SUM && lane < (int)gridDim.x) {
      // this block's part into slot blockIdx of every block of the cluster
      uint32_t a = (uint32_t)__cvta_generic_to_shared(y.red + kResWarps + y.parity * kResCluster + blockIdx.x), ra;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(lane));
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
    }
  }
  if (y.cluster) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

// The sum (SUM) over all blocks in block order; false when the bounded wait ran
// out. A part is overwritten two sums later: every block has read it by then.
template <bool SUM>
__device__ __forceinline__ bool res_wait(ResSync& y, double* sum) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x;
  if (y.cluster) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (SUM) {
      const double* s = y.red + kResWarps + y.parity * kResCluster;
      double v = 0;
      for (int i = 0; i < G; ++i) v += s[i];
      *sum = v;
    }
    return true;
  }
  if (w == 0) {
    if (lane == 0) {
      bool ok = false;
      for (int i = 0; i < y.polls && !ok; ++i) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(y.counter) : "memory");
        ok = (int)(v - y.target) >= 0;
      }
      *y.ok = ok;
    }
    __syncwarp();
    if (SUM) {
      constexpr int U = (kResMaxBlocks + 31) / 32;
      double t = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int g = 32 * u + lane;
        if (g < G) t += __ldcg(y.parts + y.parity * G + g);
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) t += __shfl_down_sync(0xffffffffu, t, s);
      if (lane == 0) y.red[kResWarps] = t;
    }
  }
  __syncthreads();
  if (SUM) *sum = y.red[kResWarps];
  return *y.ok != 0;
}

__device__ __forceinline__ void group_bar() {
  asm volatile("bar.sync %0, 128;" ::"r"((int)(threadIdx.x >> 7) + 1) : "memory");
}

// ---- level 0: a group of 128 threads per brick, thread t the z-run of four
// cells (t & 63) + 256 (t >> 6) + 64 k (as the level-0 kernels)
struct Res0 {
  int b;          // the brick
  int c0;         // its run's first cell (pool index)
  int hn[3];      // pool index of the thread's three halo cells, -1 absent
  uint16_t mk[kCPT];
};

// Halo slot of axis a of thread t and the cell's offset in the neighbour brick (halo_slot's map).
__device__ __forceinline__ void res_halo(int t, int a, int* slot, int* off) {
  const int tt = t & 63, sg = t >> 6, u = tt & 7, v = tt >> 3, e = sg ? 8 : -1, w = sg ? 0 : 7;
  if (a == 0) {
    *slot = s1(e, u, v);
    *off = w + 8 * u + 64 * v;
  } else if (a == 1) {
    *slot = s1(u, e, v);
    *off = u + 8 * w + 64 * v;
  } else {
    *slot = s1(u, v, e);
    *off = u + 8 * v + 64 * w;
  }
}

template <class T>
__device__ __forceinline__ void res0_load(const ResArgs<T>& A, int j, Res0& s) {
  const int t = threadIdx.x & 127;
  const int* row = A.drow + 8 * (size_t)j;
  s.b = row[0];
  s.c0 = s.b * kCells + (t & 63) + 256 * (t >> 6);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int slot, off;
    res_halo(t, a, &slot, &off);
    const int nb = row[1 + 2 * a + (t >> 6)];
    s.hn[a] = nb < 0 ? -1 : nb * kCells + off;
  }
#pragma unroll
  for (int k = 0; k < kCPT; ++k) s.mk[k] = A.fmask[s.c0 + 64 * k];
}

// Own run and halo values into the group's staging; the caller's next group_bar makes them readable.
template <class S>
__device__ __forceinline__ void res0_stage(S* st, const S* own, const S* halo) {
  const int t = threadIdx.x & 127;
  const int si0 = s1_of((t & 63) + 256 * (t >> 6));
#pragma unroll
  for (int k = 0; k < kCPT; ++k) st[si0 + 100 * k] = own[k];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int slot, off;
    res_halo(t, a, &slot, &off);
    st[slot] = halo[a];
  }
}

// k0_pre: finishes the previous iteration (update) and takes two sweeps from zero; returns the run's part of r.r
template <class T>
__device__ __forceinline__ double res0_pre(const ResArgs<T>& A, const Res0& s, const T* sdt, T* st, const double* rin, double* rout,
                                  const double* p, double al, int update) {
  const Params& P = A.P;
  const T om = (T)P.mgw1, om2 = (T)P.mgw2, c0 = (T)(P.mgw1 + P.mgw2 - P.mgw1 * P.mgw2);
  const T ih2[3] = {(T)P.ih2[0], (T)P.ih2[1], (T)P.ih2[2]};
  double rv[kCPT], hv[3], qv[kCPT], hq[3], xv[kCPT], pv[kCPT];
  uint16_t hm[3];
#pragma unroll
  for (int k = 0; k < kCPT; ++k) {
    rv[k] = rin[s.c0 + 64 * k];
    if (update) {
      qv[k] = A.q[s.c0 + 64 * k];
      xv[k] = A.x[s.c0 + 64 * k];
      pv[k] = p[s.c0 + 64 * k];
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int n = s.hn[a];
    hm[a] = n < 0 ? 0 : A.fmask[n];
    hv[a] = n < 0 ? 0.0 : rin[n];
    hq[a] = n < 0 || !update ? 0.0 : A.q[n];
  }
  double rr = 0;
  T own[kCPT], halo[3];
#pragma unroll
  for (int k = 0; k < kCPT; ++k) {
    if (update) {
      rv[k] = rv[k] - al * qv[k];
      rout[s.c0 + 64 * k] = rv[k];
      A.x[s.c0 + 64 * k] = xv[k] + al * pv[k];
      rr += rv[k] * rv[k];
    }
    own[k] = om * sdt[active_index(s.mk[k])] * (T)rv[k];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (update) hv[a] = hv[a] - al * hq[a];
    halo[a] = s.hn[a] < 0 ? (T)0 : om * sdt[active_index(hm[a])] * (T)hv[a];
  }
  res0_stage(st, own, halo);
  group_bar();
  const int t = threadIdx.x & 127, si0 = s1_of((t & 63) + 256 * (t >> 6));
#pragma unroll
  for (int k = 0; k < kCPT; ++k) {
    const uint16_t m = s.mk[k];
    T out = 0;
    if (m & kDomainBit) {
      const T dinv = sdt[active_index(m)];
      T sum = 0;
#pragma unroll
      for (int f = 0; f < 6; ++f)
        if (m & (1u << f)) sum += ih2[f >> 1] * zrun_nbr(st, own, si0 + 100 * k, k, f);
      out = dinv * (c0 * (T)rv[k] + om2 * sum);
    }
    A.e0[s.c0 + 64 * k] = out;
  }
  return rr;
}

// M v on cell k of the run from the staged values
template <class T, class S>
__device__ __forceinline__ S res0_apply(const S* st, const S* own, const S* ih2, uint16_t m, int si, int k) {
  S me = 0;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    if (m & (1u << (8 + f))) me += ih2[f >> 1] * own[k];
    if (m & (1u << f)) me -= ih2[f >> 1] * zrun_nbr(st, own, si, k, f);
  }
  return me;
}

template <class T>
__device__ __forceinline__ void res0_restrict(const ResArgs<T>& A, const Res0& s, T* st, const double* r) {
  const T ih2[3] = {(T)A.P.ih2[0], (T)A.P.ih2[1], (T)A.P.ih2[2]};
  T own[kCPT], halo[3], v[kCPT];
  double rk[kCPT];
#pragma unroll
  for (int k = 0; k < kCPT; ++k) {
    own[k] = A.e0[s.c0 + 64 * k];
    rk[k] = r[s.c0 + 64 * k];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) halo[a] = s.hn[a] < 0 ? (T)0 : A.e0[s.hn[a]];
  res0_stage(st, own, halo);
  group_bar();
  const int t = threadIdx.x & 127, si0 = s1_of((t & 63) + 256 * (t >> 6));
#pragma unroll
  for (int k = 0; k < kCPT; ++k)
    v[k] = (s.mk[k] & kDomainBit) ? (T)rk[k] - res0_apply<T, T>(st, own, ih2, s.mk[k], si0 + 100 * k, k) : (T)0;
  T a0 = v[0] + v[1], a1 = v[2] + v[3];
  a0 += __shfl_xor_sync(0xffffffffu, a0, 1);
  a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
  a0 += __shfl_xor_sync(0xffffffffu, a0, 8);
  a1 += __shfl_xor_sync(0xffffffffu, a1, 8);
  const int x = t & 7, y = (t >> 3) & 7, zh = t >> 6;
  if (!((x | y) & 1)) {
    const size_t base = (size_t)s.b * 64 + (x >> 1) + 4 * (y >> 1) + 16 * (2 * zh);
    A.r1[base] = a0;
    A.r1[base + 16] = a1;
  }
}

// k0_post: FIRST adds the coarse correction and writes e0b, otherwise z; returns the run's part of r.z
template <class T, bool FIRST>
__device__ __forceinline__ double res0_post(const ResArgs<T>& A, const Res0& s, const T* sdt, T* st, const double* r) {
  const T ih2[3] = {(T)A.P.ih2[0], (T)A.P.ih2[1], (T)A.P.ih2[2]}, om = (T)(FIRST ? A.P.mgw1 : A.P.mgw2);
  const T* e = FIRST ? A.e0 : A.e0b;
  T own[kCPT], halo[3];
  double rk[kCPT];
#pragma unroll
  for (int k = 0; k < kCPT; ++k) {
    own[k] = e[s.c0 + 64 * k];
    rk[k] = r[s.c0 + 64 * k];
    if (FIRST) own[k] += A.e1[(size_t)s.b * 64 + parent_off((s.c0 + 64 * k) & 511)];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int n = s.hn[a];
    halo[a] = n < 0 ? (T)0 : (FIRST ? e[n] + A.e1[(size_t)(n >> 9) * 64 + parent_off(n & 511)] : e[n]);
  }
  res0_stage(st, own, halo);
  group_bar();
  const int t = threadIdx.x & 127, si0 = s1_of((t & 63) + 256 * (t >> 6));
  double rz = 0;
#pragma unroll
  for (int k = 0; k < kCPT; ++k) {
    const uint16_t m = s.mk[k];
    T out = 0;
    if (m & kDomainBit) {
      const T me = res0_apply<T, T>(st, own, ih2, m, si0 + 100 * k, k);
      out = own[k] + om * sdt[active_index(m)] * ((T)rk[k] - me);
    }
    if (FIRST) {
      A.e0b[s.c0 + 64 * k] = out;
    } else {
      A.z[s.c0 + 64 * k] = (double)out;
      if (m & kDomainBit) rz += rk[k] * (double)out;
    }
  }
  return rz;
}

// k_update_spmv: p = z + beta p_old, q = M p; returns the run's part of p.q
template <class T>
__device__ __forceinline__ double res0_spmv(const ResArgs<T>& A, const Res0& s, double* st, const double* pold, double* pnew,
                                   double be, int first) {
  double own[kCPT], halo[3];
#pragma unroll
  for (int k = 0; k < kCPT; ++k) own[k] = A.z[s.c0 + 64 * k];
#pragma unroll
  for (int a = 0; a < 3; ++a) halo[a] = s.hn[a] < 0 ? 0.0 : A.z[s.hn[a]];
  if (!first) {
#pragma unroll
    for (int k = 0; k < kCPT; ++k) own[k] = own[k] + be * pold[s.c0 + 64 * k];
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (s.hn[a] >= 0) halo[a] = halo[a] + be * pold[s.hn[a]];
  }
  res0_stage(st, own, halo);
  group_bar();
  const int t = threadIdx.x & 127, si0 = s1_of((t & 63) + 256 * (t >> 6));
  double pq = 0;
#pragma unroll
  for (int k = 0; k < kCPT; ++k) {
    const uint16_t m = s.mk[k];
    double v = 0, p = 0;
    if (m & kDomainBit) {
      p = own[k];
      v = res0_apply<T, double>(st, own, A.P.ih2, m, si0 + 100 * k, k);
      pq += p * v;
    }
    pnew[s.c0 + 64 * k] = p;
    A.q[s.c0 + 64 * k] = v;
  }
  return pq;
}

// ---- levels 1 and 2 (D = 4, 2 cells a side per brick): the static part of a cell
template <class T>
struct ResL {
  int i;               // cell index of the level, -1: past the end
  int n[6];            // -x +x -y +y -z +z neighbours (the cell itself where absent: weight 0)
  T wl[3], wr[3], wd, dinv;
  int pc, px;          // level 1 with a dense level 2: the parent's cell there, the cell's parities (bit a: odd on axis a)
};

// CHILD: item g is child g & 7 of coarse cell g >> 3 of the list, else cell g
template <class T, int D, bool CHILD>
__device__ __forceinline__ void resl_load(const ResArgs<T>& A, int64_t g, ResL<T>& s, int& jbrick, int& o) {
  constexpr int N = D * D * D, H = D / 2;
  const T* w = D == 4 ? A.w1 : A.w2;
  const size_t ncap = D == 4 ? A.ncap1 : A.ncap2;
  s.i = -1;
  if (g >= (int64_t)A.nd * N) return;
  jbrick = (int)(g / N);
  o = (int)(g % N);
  const int* row = A.drow + 8 * (size_t)jbrick;
  int x, y, z;
  if (CHILD) {
    const int p = o >> 3, k = o & 7;
    x = 2 * (p % H) + (k & 1);
    y = 2 * ((p / H) % H) + ((k >> 1) & 1);
    z = 2 * (p / (H * H)) + (k >> 2);
  } else {
    x = o % D;
    y = (o / D) % D;
    z = o / (D * D);
  }
  const int c[3] = {x, y, z}, sd[3] = {1, D, D * D};
  const int self = x + D * y + D * D * z, i = row[0] * N + self;
  s.i = i;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int l = i - sd[a], r = i + sd[a];
    bool hr = true;
    if (c[a] == 0) {
      const int nb = row[1 + 2 * a];
      l = nb < 0 ? i : nb * N + self + (D - 1) * sd[a];
    }
    if (c[a] == D - 1) {
      const int nb = row[2 + 2 * a];
      hr = nb >= 0;
      r = hr ? nb * N + self - (D - 1) * sd[a] : i;
    }
    s.n[2 * a] = l;
    s.n[2 * a + 1] = r;
    s.wl[a] = w[a * ncap + i];
    s.wr[a] = hr ? w[a * ncap + r] : (T)0;
  }
  s.wd = w[3 * ncap + i];
  s.dinv = w[4 * ncap + i];
  if (D == 4 && A.l2) {
    const int nx = A.S.L[0].nx, ny = A.S.L[0].ny, d = row[7], yz = d / nx, bx = d - yz * nx, bz = yz / ny,
              by = yz - bz * ny;
    s.pc = (2 * bx + (x >> 1)) + 2 * nx * ((2 * by + (y >> 1)) + 2 * ny * (2 * bz + (z >> 1)));
    s.px = (x & 1) + 2 * (y & 1) + 4 * (z & 1);
  }
}

template <class T, int D>
__device__ __forceinline__ void resl_pre(const ResArgs<T>& A, const ResL<T>& s, const T* r, T* e) {
  const T* dv = (D == 4 ? A.w1 : A.w2) + 4 * (D == 4 ? A.ncap1 : A.ncap2);
  const T w1 = (T)A.P.mgw1, w2 = (T)A.P.mgw2;
  if (s.i < 0) return;
  T sum = 0;
  if (s.dinv != 0) {
    T rn[6], dn[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      rn[f] = r[s.n[f]];
      dn[f] = dv[s.n[f]];
    }
    const T rc = r[s.i];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (s.wl[a] != 0) sum += s.wl[a] * w1 * dn[2 * a] * rn[2 * a];
      if (s.wr[a] != 0) sum += s.wr[a] * w1 * dn[2 * a + 1] * rn[2 * a + 1];
    }
    sum = s.dinv * ((w1 + w2 - w1 * w2) * rc + w2 * sum);
  }
  e[s.i] = sum;
}

template <class T>
__device__ __forceinline__ T resl_apply(const ResL<T>& s, const T* ev, T ec) {
  T m = s.wd * ec;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (s.wl[a] != 0) m -= s.wl[a] * ev[2 * a];
    if (s.wr[a] != 0) m -= s.wr[a] * ev[2 * a + 1];
  }
  return m;
}

// Every lane of the warp calls it (shuffles); rc: the coarse level's residual.
template <class T, int D>
__device__ __forceinline__ void resl_restrict(const ResArgs<T>& A, const ResL<T>& s, int jbrick, int o, const T* r, const T* e,
                                     T* rc) {
  constexpr int H = D / 2;
  T v = 0;
  if (s.i >= 0 && s.dinv != 0) {
    T ev[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) ev[f] = e[s.n[f]];
    v = r[s.i] - resl_apply(s, ev, e[s.i]);
  }
  v = sum8(v);
  if (s.i >= 0 && (threadIdx.x & 7) == 0) {
    const int* row = A.drow + 8 * (size_t)jbrick;
    if (D == 2) rc[row[7]] = v;
    else if (A.l2) rc[s.pc] = v;
    else rc[(size_t)row[0] * H * H * H + (o >> 3)] = v;
  }
}

// One Jacobi sweep; COARSE adds the coarse correction first (D = 4: level 2 in
// the neighbours' bricks, D = 2: the dense level 3, whose cell of a neighbour
// brick is a stride away).
template <class T, int D, bool COARSE>
__device__ __forceinline__ void resl_jacobi(const ResArgs<T>& A, const ResL<T>& s, int jbrick, int o, const T* r, const T* e,
                                   const T* ec, T* eout) {
  constexpr int N = D * D * D, H = D / 2;
  if (s.i < 0) return;
  if (s.dinv == 0) {
    eout[s.i] = (T)0;
    return;
  }
  T ev[6], vc = e[s.i];
  const T ri = r[s.i];
#pragma unroll
  for (int f = 0; f < 6; ++f) ev[f] = e[s.n[f]];
  if (COARSE) {
    if (D == 2) {
      const DView<T>& L = A.S.L[0];
      const int n3 = (int)L.n, st[3] = {1, L.nx, L.nx * L.ny};
      const int d0 = A.drow[8 * (size_t)jbrick + 7];
      const int c[3] = {o & 1, (o >> 1) & 1, o >> 2};
      vc += ec[d0];
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        const int a = f >> 1;
        int d = d0;
        if ((f & 1) && c[a] == 1) d = d0 + st[a];
        if (!(f & 1) && c[a] == 0) d = d0 - st[a];
        ev[f] += ec[d < 0 || d >= n3 ? d0 : d];
      }
    } else if (A.l2) {
      const int nx = A.S.L[0].nx, ny = A.S.L[0].ny, n2 = 8 * (int)A.S.L[0].n, st[3] = {1, 2 * nx, 4 * nx * ny};
      vc += ec[s.pc];
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        const int a = f >> 1, odd = (s.px >> a) & 1;
        const int d = s.pc + ((f & 1) ? (odd ? st[a] : 0) : (odd ? 0 : -st[a]));
        ev[f] += ec[d < 0 || d >= n2 ? s.pc : d];  // outside the box the weight is 0
      }
    } else {
      auto par = [&](int i) -> int {
        const int q = i % N;
        return i / N * (H * H * H) + ((q % D) >> 1) + H * (((q / D) % D) >> 1) + H * H * ((q / (D * D)) >> 1);
      };
      vc += ec[par(s.i)];
#pragma unroll
      for (int f = 0; f < 6; ++f) ev[f] += ec[par(s.n[f])];
    }
  }
  const T om = (T)(COARSE ? A.P.mgw1 : A.P.mgw2);
  eout[s.i] = vc + om * s.dinv * (ri - resl_apply(s, ev, vc));
}

// ---- block 0's coarse levels, kept in shared memory for the whole solve
// A level's arrays are padded with zeros so that a sweep reads a cell's six
// neighbours at fixed strides without asking where it lies: the face weights
// over the grid's edge are 0 (Galerkin weights of faces without a cell behind
// them), and the values there are the padding or the next row's, finite.
template <class T>
struct BL {
  int nx, ny, nz, n;
  T *e, *e2, *r;          // n cells and nx ny zeros on either side
  T *w;                   // left-face weights x, y, z: three runs of n + nx ny
  T *wd, *dinv;           // diagonal; its inverse, padded as e
  uint16_t* par;          // the parent's cell on the next level
};
constexpr int kResBlk = kMaxDense + 1;

__host__ __device__ inline size_t bl_bytes(int64_t n, int64_t plane, size_t ts) {
  return (ts * (size_t)(4 * (n + 2 * plane) + 3 * (n + plane) + n) + 2 * (size_t)n + 15) / 16 * 16;
}
template <class T>
__device__ inline unsigned char* bl_carve(BL<T>& L, unsigned char* p, int nx, int ny, int nz) {
  const int n = nx * ny * nz, pl = nx * ny;
  L.nx = nx;
  L.ny = ny;
  L.nz = nz;
  L.n = n;
  T* t = reinterpret_cast<T*>(p);
  L.e = t + pl;
  L.e2 = L.e + n + 2 * pl;
  L.r = L.e2 + n + 2 * pl;
  L.dinv = L.r + n + 2 * pl;
  L.w = L.dinv + n + pl;
  L.wd = L.w + 3 * (n + pl);
  L.par = reinterpret_cast<uint16_t*>(L.wd + n);
  return p + bl_bytes(n, pl, sizeof(T));
}

// Two sweeps from zero, as kl_pre.
template <class T>
__device__ inline void bl_pre(const BL<T>& L, T w1, T w2) {
  const int n = L.n, pl = L.nx * L.ny, st[3] = {1, L.nx, pl};
  for (int i = threadIdx.x; i < n; i += kResThreads) {
    T s = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const T* w = L.w + a * (n + pl) + i;
      s += w[0] * w1 * L.dinv[i - st[a]] * L.r[i - st[a]];
      s += w[st[a]] * w1 * L.dinv[i + st[a]] * L.r[i + st[a]];
    }
    L.e[i] = L.dinv[i] * ((w1 + w2 - w1 * w2) * L.r[i] + w2 * s);
  }
}
// RESIDUAL: out = r - M e (0 off the domain), else one Jacobi sweep.
template <class T, bool RESIDUAL>
__device__ inline void bl_sweep(const BL<T>& L, const T* e, T* out, T om) {
  const int n = L.n, pl = L.nx * L.ny, st[3] = {1, L.nx, pl};
  for (int i = threadIdx.x; i < n; i += kResThreads) {
    const T ec = e[i], di = L.dinv[i];
    T s = L.wd[i] * ec;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const T* w = L.w + a * (n + pl) + i;
      s -= w[0] * e[i - st[a]];
      s -= w[st[a]] * e[i + st[a]];
    }
    const T v = L.r[i] - s;
    out[i] = di == 0 ? (T)0 : (RESIDUAL ? v : ec + om * di * v);
  }
}

template <class T>
__device__ inline void res_coarse(const BL<T>* L, int nl, const T* rin, T* eout, T w1, T w2, const double* sinv,
                                  bool exact) {
  for (int i = threadIdx.x; i < L[0].n; i += kResThreads) L[0].r[i] = L[0].dinv[i] == 0 ? (T)0 : rin[i];
  __syncthreads();
  for (int l = 0; l + 1 < nl; ++l) {
    const BL<T>&F = L[l], &C = L[l + 1];
    bl_pre(F, w1, w2);
    __syncthreads();
    bl_sweep<T, true>(F, F.e, F.e2, (T)0);
    __syncthreads();
    const float rnx = 1.0f / (float)C.nx, rny = 1.0f / (float)C.ny;
    for (int I = threadIdx.x; I < C.n; I += kResThreads) {
      const int xy = qdiv(I, C.nx, rnx), X = I - xy * C.nx, Z = qdiv(xy, C.ny, rny), Y = xy - Z * C.ny;
      T s = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int x = 2 * X + (k & 1), y = 2 * Y + ((k >> 1) & 1), z = 2 * Z + (k >> 2);
        if (x < F.nx && y < F.ny && z < F.nz) s += F.e2[x + F.nx * (y + F.ny * z)];
      }
      C.r[I] = s;
    }
    __syncthreads();
  }
  const BL<T>& B = L[nl - 1];
  if (exact) {
    // row i of inv r by 16 lanes
    const int n = B.n, p = threadIdx.x & 15;
    for (int i = threadIdx.x >> 4; i < (n + 1) / 2 * 2; i += kResThreads / 16) {
      double s = 0.0;
      if (i < n)
        for (int j = p; j < n; j += 16) s += sinv[i * 64 + j] * (double)B.r[j];
#pragma unroll
      for (int m = 8; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m, 16);
      if (i < n && p == 0) B.e[i] = B.dinv[i] == 0 ? (T)0 : (T)s;
    }
    __syncthreads();
  } else {
    bl_pre(B, w1, w2);
    __syncthreads();
    for (int s = 2; s < kCoarsestSweeps; s += 2) {
      bl_sweep<T, false>(B, B.e, B.e2, w1);
      __syncthreads();
      bl_sweep<T, false>(B, B.e2, B.e, w2);
      __syncthreads();
    }
  }
  for (int l = nl - 2; l >= 0; --l) {
    const BL<T>&F = L[l], &C = L[l + 1];
    for (int i = threadIdx.x; i < F.n; i += kResThreads) F.e[i] += C.e[F.par[i]];
    __syncthreads();
    bl_sweep<T, false>(F, F.e, F.e2, w1);
    __syncthreads();
    bl_sweep<T, false>(F, F.e2, F.e, w2);
    __syncthreads();
  }
  for (int i = threadIdx.x; i < L[0].n; i += kResThreads) eout[i] = L[0].e[i];
}

// Carves and fills block 0's levels (static for the solve); returns their number.
template <class T>
__device__ inline int res_coarse_init(const ResArgs<T>& A, BL<T>* L, unsigned char* smem, size_t bytes) {
  const int nl = A.S.hi + (A.l2 ? 1 : 0);
  if (threadIdx.x == 0) {
    unsigned char* p = smem;
    int k = 0;
    if (A.l2) p = bl_carve(L[k++], p, 2 * A.S.L[0].nx, 2 * A.S.L[0].ny, 2 * A.S.L[0].nz);
    for (int l = 0; l < A.S.hi; ++l) p = bl_carve(L[k++], p, A.S.L[l].nx, A.S.L[l].ny, A.S.L[l].nz);
  }
  for (size_t i = threadIdx.x; i < bytes / 16; i += kResThreads)
    reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  if (A.l2) {
    const BL<T>& F = L[0];
    const int nx = A.S.L[0].nx, ny = A.S.L[0].ny, pl = F.nx * F.ny;
    for (int g = threadIdx.x; g < 8 * A.nd; g += kResThreads) {
      const int* row = A.drow + 8 * (size_t)(g >> 3);
      const int o = g & 7, d = row[7], yz = d / nx, bx = d - yz * nx, bz = yz / ny, by = yz - bz * ny;
      const int i = (2 * bx + (o & 1)) + F.nx * ((2 * by + ((o >> 1) & 1)) + F.ny * (2 * bz + (o >> 2)));
      const size_t q = (size_t)row[0] * 8 + o;
      for (int a = 0; a < 3; ++a) F.w[a * (F.n + pl) + i] = A.w2[a * A.ncap2 + q];
      F.wd[i] = A.w2[3 * A.ncap2 + q];
      F.dinv[i] = A.w2[4 * A.ncap2 + q];
    }
  }
  for (int l = 0; l < A.S.hi; ++l) {
    const BL<T>& F = L[l + (A.l2 ? 1 : 0)];
    const T* w = A.S.L[l].w;
    const int pl = F.nx * F.ny;
    for (int i = threadIdx.x; i < F.n; i += kResThreads) {
      for (int a = 0; a < 3; ++a) F.w[a * (F.n + pl) + i] = w[(size_t)a * F.n + i];
      F.wd[i] = w[(size_t)3 * F.n + i];
      F.dinv[i] = w[(size_t)4 * F.n + i];
    }
  }
  for (int k = 0; k + 1 < nl; ++k) {
    const BL<T>&F = L[k], &C = L[k + 1];
    for (int i = threadIdx.x; i < F.n; i += kResThreads) {
      const int x = i % F.nx, y = (i / F.nx) % F.ny, z = i / (F.nx * F.ny);
      F.par[i] = (uint16_t)((x >> 1) + C.nx * ((y >> 1) + C.ny * (z >> 1)));
    }
  }
  __syncthreads();
  return nl;
}

// Shared memory of a block: the groups' staging and, in block 0, the coarse
// levels and the coarsest inverse.
constexpr int kResStage = kResGroups * kS1 * 8;
constexpr int kResInv = 64 * 64 * 8;

template <class T>
__global__ void __launch_bounds__(kResThreads, 1) k_cg_resident(const __grid_constant__ ResArgs<T> A) {
  extern __shared__ __align__(128) unsigned char res_smem[];
  __shared__ BL<T> SL[kResBlk];
  __shared__ double red[kResWarps + 2 * kResCluster + 2];
  __shared__ int sok;
  // the inverse diagonals by face count: lanes of a warp index it apart, which
  // the constant bank of the kernel's parameters would serve one by one
  __shared__ T sdt[27];
  if (threadIdx.x < 27) sdt[threadIdx.x] = (T)A.P.dtab[threadIdx.x];
  double* st64 = reinterpret_cast<double*>(res_smem) + (threadIdx.x >> 7) * kS1;
  T* st = reinterpret_cast<T*>(st64);
  Scalars* ds = A.ds;
  // After a wait that ran out the count of arrivals is off until the next upload
  // clears it together with the mark. One thread asks: a block of this launch may
  // set the mark meanwhile.
  if (threadIdx.x == 0) sok = ds->done || (ds->err & kErrTimeout);
  __syncthreads();
  if (sok) return;
  const int nd = A.nd, G = gridDim.x;
  const T w1 = (T)A.P.mgw1, w2 = (T)A.P.mgw2;
  double* sinv = reinterpret_cast<double*>(res_smem + kResStage);
  bool exact = false;
  int nl = 0;
  if (blockIdx.x == 0) {
    nl = res_coarse_init(A, SL, res_smem + kResStage + kResInv, A.blk_bytes);
    exact = *A.inv_ok && SL[nl - 1].n <= 64;
    if (exact) blk_copy(sinv, A.inv, (int64_t)SL[nl - 1].n * 64);
  }
  // the count goes on from the last solve's, so nothing is cleared: what it was
  // then is kept beside it (block 0 writes it once every block has read it). Blocks
  // that give up leave at different counts: no solve starts from there (above).
  unsigned* counter = reinterpret_cast<unsigned*>(A.slots);
  unsigned* last = counter + 32;
  __syncthreads();
  ResSync y{counter, reinterpret_cast<double*>(A.slots + 32), *last, 0u, A.cluster, A.polls, red, &sok};
  // bricks by group and cells by warp, dealt to the blocks in turn, so that a
  // system smaller than the grid still spreads over every SM
  const int j0 = (threadIdx.x >> 7) * G + blockIdx.x, dj = G * kResGroups;
  const int64_t g0 = ((int64_t)(threadIdx.x >> 5) * G + blockIdx.x) * 32 + (threadIdx.x & 31),
                dg = (int64_t)G * kResThreads;
  const int64_t n1 = (int64_t)nd * 64, n2 = (int64_t)nd * 8;
  double *r = A.r, *rn = A.r2, *pd = A.pd, *pd2 = A.pd2;
  double rz = 0, rr = ds->rr, alpha = 0, beta = 0, sum = 0, dummy;
  const double bnorm2 = ds->bnorm2;
  int iters = ds->iters, first = 1, done = 0;
  bool ok = true;
  Res0 s0;
  ResL<T> sl;
  int jb = 0, o = 0;
  if (j0 < nd) res0_load(A, j0, s0);
  auto each_brick = [&](auto&& f) {
    for (int j = j0; j < nd; j += dj) {
      if (j != j0 || nd > dj) {
        if (j != j0) group_bar();  // the staging is read out
        res0_load(A, j, s0);
      }
      f();
    }
  };
#define RES_SYNC()                      \
  res_arrive<false>(y, 0.0);            \
  ok = res_wait<false>(y, &dummy) && ok; \
  if (!ok) break
  while (true) {
    // ---- the first kernel of a V-cycle, with the previous iteration's update
    sum = 0;
    const int update = first ? 0 : 1;
    each_brick([&] { sum += res0_pre(A, s0, sdt, st, r, rn, pd, alpha, update); });
    if (update) {
      double* t = r;
      r = rn;
      rn = t;
    }
    res_arrive<true>(y, sum);
    ok = res_wait<true>(y, &sum);
    if (!ok) break;
    if (update) {
      rr = sum;
      ++iters;
      if (rr <= A.rtol2 * bnorm2 || iters >= A.max_iters || !(rr == rr)) {
        done = 1;
        break;
      }
    }
    each_brick([&] { res0_restrict(A, s0, st, r); });
    res_arrive<false>(y, 0.0);
    resl_load<T, 4, false>(A, g0, sl, jb, o);
    ok = res_wait<false>(y, &dummy);
    if (!ok) break;
    // ---- levels 1 and 2 down
    for (int64_t g = g0; g < n1; g += dg) {
      if (g != g0) resl_load<T, 4, false>(A, g, sl, jb, o);
      resl_pre<T, 4>(A, sl, A.r1, A.e1);
    }
    res_arrive<false>(y, 0.0);
    resl_load<T, 4, true>(A, g0, sl, jb, o);
    ok = res_wait<false>(y, &dummy);
    if (!ok) break;
    for (int64_t g = g0; (g & ~31ll) < n1; g += dg) {
      if (g != g0) resl_load<T, 4, true>(A, g, sl, jb, o);
      resl_restrict<T, 4>(A, sl, jb, o, A.r1, A.e1, A.r2l);
    }
    if (!A.l2) {
      res_arrive<false>(y, 0.0);
      resl_load<T, 2, false>(A, g0, sl, jb, o);
      ok = res_wait<false>(y, &dummy);
      if (!ok) break;
      for (int64_t g = g0; g < n2; g += dg) {
        if (g != g0) resl_load<T, 2, false>(A, g, sl, jb, o);
        resl_pre<T, 2>(A, sl, A.r2l, A.e2);
      }
      res_arrive<false>(y, 0.0);
      resl_load<T, 2, true>(A, g0, sl, jb, o);
      ok = res_wait<false>(y, &dummy);
      if (!ok) break;
      for (int64_t g = g0; (g & ~31ll) < n2; g += dg) {
        if (g != g0) resl_load<T, 2, true>(A, g, sl, jb, o);
        resl_restrict<T, 2>(A, sl, jb, o, A.r2l, A.e2, A.S.L[0].r);
      }
    }
    RES_SYNC();
    // ---- level 3 and below (and level 2) by block 0
    if (blockIdx.x == 0)
      res_coarse(SL, nl, A.l2 ? A.r2l : A.S.L[0].r, A.l2 ? A.e2 : A.S.L[0].e, w1, w2, sinv, exact);
    if (A.l2) {
      res_arrive<false>(y, 0.0);
      resl_load<T, 4, false>(A, g0, sl, jb, o);
      ok = res_wait<false>(y, &dummy);
      if (!ok) break;
    } else {
      RES_SYNC();
      // ---- level 2 up
      resl_load<T, 2, false>(A, g0, sl, jb, o);
      for (int64_t g = g0; g < n2; g += dg) {
        if (g != g0) resl_load<T, 2, false>(A, g, sl, jb, o);
        resl_jacobi<T, 2, true>(A, sl, jb, o, A.r2l, A.e2, A.S.L[0].e, A.e2b);
      }
      res_arrive<false>(y, 0.0);
      if (n2 > dg) resl_load<T, 2, false>(A, g0, sl, jb, o);
      ok = res_wait<false>(y, &dummy);
      if (!ok) break;
      for (int64_t g = g0; g < n2; g += dg) {
        if (g != g0) resl_load<T, 2, false>(A, g, sl, jb, o);
        resl_jacobi<T, 2, false>(A, sl, jb, o, A.r2l, A.e2b, (const T*)nullptr, A.e2);
      }
      res_arrive<false>(y, 0.0);
      resl_load<T, 4, false>(A, g0, sl, jb, o);
      ok = res_wait<false>(y, &dummy);
      if (!ok) break;
    }
    // ---- level 1 up
    for (int64_t g = g0; g < n1; g += dg) {
      if (g != g0) resl_load<T, 4, false>(A, g, sl, jb, o);
      resl_jacobi<T, 4, true>(A, sl, jb, o, A.r1, A.e1, A.e2, A.e1b);
    }
    res_arrive<false>(y, 0.0);
    if (n1 > dg) resl_load<T, 4, false>(A, g0, sl, jb, o);
    ok = res_wait<false>(y, &dummy);
    if (!ok) break;
    for (int64_t g = g0; g < n1; g += dg) {
      if (g != g0) resl_load<T, 4, false>(A, g, sl, jb, o);
      resl_jacobi<T, 4, false>(A, sl, jb, o, A.r1, A.e1b, (const T*)nullptr, A.e1);
    }
    RES_SYNC();
    each_brick([&] { res0_post<T, true>(A, s0, sdt, st, r); });
    RES_SYNC();
    sum = 0;
    each_brick([&] { sum += res0_post<T, false>(A, s0, sdt, st, r); });
    res_arrive<true>(y, sum);
    ok = res_wait<true>(y, &sum);
    if (!ok) break;
    beta = first ? 0.0 : (rz != 0 ? sum / rz : 0.0);
    rz = sum;
    // ---- direction and product
    {
      double* t = pd;
      pd = pd2;
      pd2 = t;
    }
    sum = 0;
    each_brick([&] { sum += res0_spmv(A, s0, st64, pd2, pd, beta, first); });
    res_arrive<true>(y, sum);
    ok = res_wait<true>(y, &sum);
    if (!ok) break;
    alpha = sum != 0 ? rz / sum : 0.0;
    first = 0;
  }
#undef RES_SYNC
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    ds->rr = rr;
    ds->iters = iters;
    ds->rz = rz;
    ds->alpha = alpha;
    ds->beta = beta;
    ds->done = done;
    if (!A.cluster) *last = y.target;
  }
  if (!ok && threadIdx.x == 0) atomicOr(&ds->err, kErrTimeout);
  // no block of a cluster leaves while another may still write its slots
  if (A.cluster) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// Systems of at most this many domain bricks go to one cluster of at most
// kResCluster blocks. The cluster is the faster one up to a brick a group (us an
// iteration, FP64, cluster and grid: 48 bricks 26 and 30, 64 29 and 30; FP32 levels 24
// and 28, 25 and 28); with a second round of bricks the grid is (72: 39 and 33, 108: 43
// and 34; FP32 34 and 31, 37 and 31). The line stays at two rounds all the same: the
// forms add their dot products in other orders, and with FP32 levels the pressures of
// systems between the lines would move by more than 1e-9 of themselves, inside the
// solve's tolerance but not reproducibly with earlier results.
constexpr int kResClusterBricks = 128;
// Level 2 joins block 0's levels up to this many cells (ms a projection, with it and
// with level 2 spread over the blocks: 18 bricks of a 3 x 3 x 3 box 0.43 and 0.50, 512
// of 8 x 8 x 8 (4,096 cells) 0.93 and 0.94; past the line, 490 of 9 x 9 x 9, 0.94 and
// 0.89).
constexpr int kResBlk2 = 4096;

template <class T>
static int cg_resident_t(Ctx* c, int* enqueued) {
  size_t blk = 0;
  for (int l = 0; l < c->ndense; ++l)
    blk += bl_bytes(c->dense[l].n, (int64_t)c->dense[l].nx * c->dense[l].ny, sizeof(T));
  const size_t room = (size_t)c->res_smem;
  if (kResStage + kResInv + blk > room || c->dense[0].n > 65535) return MAC_OK;
  // level 2 joins block 0's levels when it fits beside them: four exchanges
  // fewer a V-cycle, against sweeps by one block (up to kResBlk2 cells)
  const int64_t n2 = 8 * c->dense[0].n;
  const size_t b2 = bl_bytes(n2, 4 * (int64_t)c->dense[0].nx * c->dense[0].ny, sizeof(T));
  const int l2 = n2 <= kResBlk2 && c->dense[0].n <= c->cap_bricks && kResStage + kResInv + blk + b2 <= room;
  if (l2) blk += b2;
  const size_t smem = kResStage + kResInv + blk;
  const int nd = c->ndom_host;
  ResArgs<T> A;
  A.drow = c->drow;
  A.nd = nd;
  A.fmask = c->fmask;
  A.r = c->r;
  A.r2 = c->r2;
  A.x = c->x;
  A.pd = c->pd;
  A.pd2 = c->pd2;
  A.q = c->q;
  A.z = c->z;
  A.e0 = (T*)c->mg_e[0];
  A.e0b = (T*)c->mg_e2[0];
  A.e1 = (T*)c->mg_e[1];
  A.e1b = (T*)c->mg_e2[1];
  A.e2 = (T*)c->mg_e[2];
  A.e2b = (T*)c->mg_e2[2];
  A.r1 = (T*)c->mg_r[1];
  A.r2l = (T*)c->mg_r[2];
  A.w1 = (const T*)c->mg_w[1];
  A.w2 = (const T*)c->mg_w[2];
  A.ncap1 = (size_t)c->cap_bricks * 64;
  A.ncap2 = (size_t)c->cap_bricks * 8;
  for (int l = 0; l < c->ndense; ++l) A.S.L[l] = dview<T>(c, l);
  A.l2 = l2;
  A.blk_bytes = blk;
  A.S.lo = 0;
  A.S.hi = c->ndense;
  A.inv = c->coarse_inv;
  A.inv_ok = c->coarse_ok;
  A.ds = c->ds;
  A.slots = c->res_slots;
  A.P = c->dp;
  A.rtol2 = c->prm.rtol * c->prm.rtol;
  A.max_iters = c->prm.max_iters;
  A.polls = c->wait_polls;
  A.cluster = nd <= kResClusterBricks && c->res_cluster ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.blockDim = kResThreads;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (A.cluster) {
    int g = 1;
    while (g < kResCluster && g * kResGroups < nd) g *= 2;
    cfg.gridDim = g;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = g;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    cfg.gridDim = nd < c->res_grid ? nd : c->res_grid;
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  void* args[] = {&A};
  launch_resident(cfg, (const void*)k_cg_resident<T>, args, enqueued);
  if (*enqueued) MAC_COUNT(c);
  return MAC_OK;
}

// Enqueues the whole CG loop of a multigrid form as one kernel when the system
// is of a size for it; otherwise *enqueued = 0 and nothing is launched. The
// line is where level 3 (a cell per brick of the domain's box) is a level for
// one block (mac_set_coarse_block): beyond it, its sweeps need exchanges of
// their own and the bricks several rounds a phase, and the launches are no
// slower (2,100 bricks, FP64: 112 against 118 us an iteration; a sparse box of
// 27,648 cells: 92 against 75). Other sweep counts and the prefetching first
// kernel keep the launches.
int cg_resident(Ctx* c, int* enqueued) {
  *enqueued = 0;
  if (c->mg_sweeps0 != 2 || c->mg_bulk || c->res_grid < 1 || c->dense[0].n > c->blk_max_cells) return MAC_OK;
  return c->mg_float ? cg_resident_t<float>(c, enqueued) : cg_resident_t<double>(c, enqueued);
}

// What a device offers the resident form: its blocks (one an SM), dynamic
// shared memory, and whether a cluster of kResCluster blocks fits. Asked once a
// device (the questions take half a millisecond, and a context is made for each
// world). The kernel's attributes are set for each context: a reset of the device
// by the host program takes them back.
struct ResDevice {
  int asked = 0, grid = 0, smem = 0, cluster = 0;
};

template <class T>
static int res_allow(int smem) {
  int rc = check(cudaFuncSetAttribute(k_cg_resident<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  return rc ? rc : check(cudaFuncSetAttribute(k_cg_resident<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

template <class T>
static int res_ask(ResDevice& d, int dev, int nsm, int optin) {
  cudaFuncAttributes fa;
  int rc = check(cudaFuncGetAttributes(&fa, k_cg_resident<T>));
  if (rc) return rc;
  d.smem = optin - (int)fa.sharedSizeBytes;
  rc = res_allow<T>(d.smem);
  int occ = 0, coop = 0, ncl = 0;
  if (!rc) rc = check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_cg_resident<T>, kResThreads, d.smem));
  if (!rc) rc = check(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (rc) return rc;
  d.grid = occ < 1 || !coop ? 0 : (nsm < kResMaxBlocks ? nsm : kResMaxBlocks);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.gridDim = kResCluster;
  cfg.blockDim = kResThreads;
  cfg.dynamicSmemBytes = d.smem;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kResCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  d.cluster = cudaOccupancyMaxActiveClusters(&ncl, k_cg_resident<T>, &cfg) == cudaSuccess && ncl > 0;
  if (!d.cluster) cudaGetLastError();
  d.asked = 1;
  return MAC_OK;
}

template <class T>
static int res_configure_t(Ctx* c, int nsm, int optin) {
  constexpr int kDevices = 64;
  static std::mutex mu;
  static ResDevice known[kDevices];
  ResDevice own, *d = &own;
  std::lock_guard<std::mutex> lock(mu);
  if (c->prm.device < kDevices) d = &known[c->prm.device];
  int rc = d->asked ? res_allow<T>(d->smem) : res_ask<T>(*d, c->prm.device, nsm, optin);
  if (rc) return rc;
  c->res_grid = d->grid;
  c->res_smem = d->smem;
  c->res_cluster = d->cluster;
  return MAC_OK;
}

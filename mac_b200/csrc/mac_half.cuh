// Level-0 stencil passes of the pressure solve by half bricks, one warp each.
//
// A warp holds a brick's lower or upper four z-planes: lane l the x-pair of
// cells 2 l, 2 l + 1 of each plane (row l / 4, pair l % 4), so a plane is one
// coalesced load of pairs. A cell's x and y neighbours come from other lanes by
// shuffles, its z neighbours from the lane's own registers, and the halo from
// eight values a lane (two x-face cells, a y-face pair, the pairs above and
// below) spread by shuffles. No shared memory and no barrier: a 10^3 array
// staged there kept that pipe 70-90% busy (two-way conflicts of its rows of
// ten, a store and four loads a cell) at 40% of the memory bandwidth. The
// arithmetic of a cell is that of the staged form. Quarter bricks a warp (twice
// the threads, more of the halo read twice) were 2.6% slower a step at 15,700
// bricks and no faster at 2,100.
#pragma once
#include "mac_internal.cuh"

namespace mac {

constexpr int kHT = 256;              // threads of a block of the half-brick kernels
constexpr int kHB = kHT / 64;         // bricks of such a block
constexpr uint32_t kFullPair = 0xBF3FBF3Fu;  // two cells in the domain with six coupled faces

inline int half_blocks(int nd) { return (nd + kHB - 1) / kHB; }

// Pool indices fit an int: a brick takes over 60 KB of a context's arrays.
struct Half {
  int b;       // the brick
  int c;       // the lane's pair of the first plane (plane k: + 64 k)
  int x;       // x halo: this cell and the one two planes up; -1 absent (also below)
  int y;       // y halo: a pair
  int zm, zp;  // the pairs below the first and above the last plane
};

// Half h (planes 4 h ..) of the brick of domain row `row`. Halo: lanes 0..15
// take the sign - faces and 16..31 the + faces; the x cell of lane l is that of
// row l & 7 on plane (l >> 3) & 1, the y pair that of plane (l >> 2) & 3.
__device__ __forceinline__ void half_load(const int* __restrict__ row, int h, Half& s) {
  const int l = threadIdx.x & 31, sg = l >> 4, z0 = 256 * h;
  const int nx = row[1 + sg], ny = row[3 + sg], nm = h == 0 ? row[5] : -1, np = h == 1 ? row[6] : -1;
  s.b = row[0];
  s.c = s.b * kCells + z0 + 2 * l;
  s.x = nx < 0 ? -1 : nx * kCells + z0 + 64 * ((l >> 3) & 1) + 8 * (l & 7) + (sg ? 0 : 7);
  s.y = ny < 0 ? -1 : ny * kCells + z0 + 64 * ((l >> 2) & 3) + 2 * (l & 3) + (sg ? 0 : 56);
  s.zm = h > 0 ? s.c - 64 : (nm < 0 ? -1 : nm * kCells + 448 + 2 * l);
  s.zp = h == 0 ? s.c + 256 : (np < 0 ? -1 : np * kCells + 2 * l);
}

__device__ __forceinline__ void half_masks(const uint16_t* fmask, const Half& s, uint32_t (&mk)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) mk[k] = *reinterpret_cast<const uint32_t*>(fmask + s.c + 64 * k);
}
__device__ __forceinline__ bool half_full(const uint32_t (&mk)[4]) {
  uint32_t m = mk[0];
#pragma unroll
  for (int k = 1; k < 4; ++k) m &= mk[k];
  return __all_sync(0xffffffffu, m == kFullPair);
}
__device__ __forceinline__ uint16_t half_mask(const uint32_t (&mk)[4], int k, int j) { return (uint16_t)(mk[k] >> (16 * j)); }

__device__ __forceinline__ void ld2(const double* p, double* v) {
  const double2 a = *reinterpret_cast<const double2*>(p);
  v[0] = a.x;
  v[1] = a.y;
}
__device__ __forceinline__ void ld2(const float* p, float* v) {
  const float2 a = *reinterpret_cast<const float2*>(p);
  v[0] = a.x;
  v[1] = a.y;
}
__device__ __forceinline__ void st2(double* p, double a, double b) { *reinterpret_cast<double2*>(p) = make_double2(a, b); }
__device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }

// Halo values of a lane: x on planes (0, 1) and (2, 3), the y pair, the pairs below and above.
template <class V>
struct HaloV {
  V x[2], y[2], m[2], p[2];
};

// one(i): the value of cell i; two(i, v): those of cells i and i + 1. Absent: 0.
template <class V, class F1, class F2>
__device__ __forceinline__ void half_halo(const Half& s, HaloV<V>& h, F1 one, F2 two) {
#pragma unroll
  for (int i = 0; i < 2; ++i) h.x[i] = (V)0;
  h.y[0] = h.y[1] = h.m[0] = h.m[1] = h.p[0] = h.p[1] = (V)0;
  if (s.x >= 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) h.x[i] = one(s.x + 128 * i);
  }
  if (s.y >= 0) two(s.y, h.y);
  if (s.zm >= 0) two(s.zm, h.m);
  if (s.zp >= 0) two(s.zp, h.p);
}

// f(k, j, nb) for every cell (plane k, pair element j) with its neighbours -x +x -y +y -z +z.
template <class V, class F>
__device__ __forceinline__ void half_each(const V (&v)[4][2], const HaloV<V>& h, F f) {
  const int l = threadIdx.x & 31, px = l & 3, y = l >> 2;
  const int sx = (px == 3 ? 16 : 0) + y, sy = (y == 7 ? 16 : 0) + px;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const V hx = __shfl_sync(0xffffffffu, h.x[k >> 1], sx + 8 * (k & 1));
    const V xl = __shfl_up_sync(0xffffffffu, v[k][1], 1), xr = __shfl_down_sync(0xffffffffu, v[k][0], 1);
    V nb[2][6];
    nb[0][0] = px == 0 ? hx : xl;
    nb[0][1] = v[k][1];
    nb[1][0] = v[k][0];
    nb[1][1] = px == 3 ? hx : xr;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const V hy = __shfl_sync(0xffffffffu, h.y[j], sy + 4 * k);
      const V yl = __shfl_up_sync(0xffffffffu, v[k][j], 4), yr = __shfl_down_sync(0xffffffffu, v[k][j], 4);
      nb[j][2] = y == 0 ? hy : yl;
      nb[j][3] = y == 7 ? hy : yr;
      nb[j][4] = k > 0 ? v[k > 0 ? k - 1 : 0][j] : h.m[j];
      nb[j][5] = k < 3 ? v[k < 3 ? k + 1 : k][j] : h.p[j];
      f(k, j, nb[j]);
    }
  }
}

// M v of a cell of face classes m
template <bool FULL, class V>
__device__ __forceinline__ V half_apply(uint16_t m, V own, const V* nb, const V* ih2) {
  V me = 0;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    if (FULL || (m & (1u << (8 + f)))) me += ih2[f >> 1] * own;
    if (FULL || (m & (1u << f))) me -= ih2[f >> 1] * nb[f];
  }
  return me;
}

// Pre-smoothing (k0_pre). dinv(m): inverse diagonal of face classes m.
template <class T, class DI>
__device__ __forceinline__ double half_pre(const Half& s, const uint32_t (&mk)[4], const uint16_t* fmask, DI dinv,
                                           const Params& P, const double* rin, double* rout, double* x,
                                           const double* p, const double* q, double al, int update, T* e) {
  const T om = (T)P.mgw1, om2 = (T)P.mgw2, c0 = (T)(P.mgw1 + P.mgw2 - P.mgw1 * P.mgw2);
  const T ih2[3] = {(T)P.ih2[0], (T)P.ih2[1], (T)P.ih2[2]};
  HaloV<T> hv;
  half_halo(
      s, hv,
      [&](int i) {
        const double v = update ? rin[i] - al * q[i] : rin[i];
        return om * dinv(fmask[i]) * (T)v;
      },
      [&](int i, T* o) {
        double v[2];
        ld2(rin + i, v);
        if (update) {
          double w[2];
          ld2(q + i, w);
          v[0] = v[0] - al * w[0];
          v[1] = v[1] - al * w[1];
        }
        const uint32_t m = *reinterpret_cast<const uint32_t*>(fmask + i);
        o[0] = om * dinv((uint16_t)m) * (T)v[0];
        o[1] = om * dinv((uint16_t)(m >> 16)) * (T)v[1];
      });
  T rv[4][2], own[4][2];
  double rr = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = s.c + 64 * k;
    double v[2];
    ld2(rin + c, v);
    if (update) {
      double w[2], xv[2], pv[2];
      ld2(q + c, w);
      ld2(x + c, xv);
      ld2(p + c, pv);
      v[0] = v[0] - al * w[0];
      v[1] = v[1] - al * w[1];
      st2(rout + c, v[0], v[1]);
      st2(x + c, xv[0] + al * pv[0], xv[1] + al * pv[1]);
      rr += v[0] * v[0];
      rr += v[1] * v[1];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      rv[k][j] = (T)v[j];
      own[k][j] = om * dinv(half_mask(mk, k, j)) * (T)v[j];
    }
  }
  T out[2] = {};
  auto put = [&](int k, int j) {
    if (j == 1) st2(e + s.c + 64 * k, out[0], out[1]);
  };
  if (half_full(mk)) {
    const T di = dinv((uint16_t)kFullPair);
    half_each(own, hv, [&](int k, int j, const T* nb) {
      T sum = 0;
#pragma unroll
      for (int f = 0; f < 6; ++f) sum += ih2[f >> 1] * nb[f];
      out[j] = di * (c0 * rv[k][j] + om2 * sum);
      put(k, j);
    });
  } else {
    half_each(own, hv, [&](int k, int j, const T* nb) {
      const uint16_t m = half_mask(mk, k, j);
      T sum = 0;
#pragma unroll
      for (int f = 0; f < 6; ++f)
        if (m & (1u << f)) sum += ih2[f >> 1] * nb[f];
      out[j] = (m & kDomainBit) ? dinv(m) * (c0 * rv[k][j] + om2 * sum) : (T)0;
      put(k, j);
    });
  }
  return rr;
}

// The lane's level-1 cell of its planes 0 and 1 (planes 2 and 3: + 16), shared with its row's other parity
__device__ __forceinline__ int half_parent(int h) {
  const int l = threadIdx.x & 31;
  return (l & 3) + 4 * (l >> 3) + 32 * h;
}

// r - M e summed over 2x2x2 children into level 1 (k0_restrict).
template <class T>
__device__ __forceinline__ void half_restrict(const Half& s, int h, const uint32_t (&mk)[4], const Params& P, const T (&own)[4][2],
                                              const HaloV<T>& hv, const double (&r)[4][2], T* r1) {
  const T ih2[3] = {(T)P.ih2[0], (T)P.ih2[1], (T)P.ih2[2]};
  T v[4][2];
  if (half_full(mk)) {
    half_each(own, hv, [&](int k, int j, const T* nb) {
      v[k][j] = (T)r[k][j] - half_apply<true>((uint16_t)0, own[k][j], nb, ih2);
    });
  } else {
    half_each(own, hv, [&](int k, int j, const T* nb) {
      const uint16_t m = half_mask(mk, k, j);
      const T a = half_apply<false>(m, own[k][j], nb, ih2);
      v[k][j] = (m & kDomainBit) ? (T)r[k][j] - a : (T)0;
    });
  }
  // z pairs and x pairs are the lane's own, the y pair is in lanes l, l ^ 4
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const T a = v[2 * q][0] + v[2 * q + 1][0], b = v[2 * q][1] + v[2 * q + 1][1];
    T t = a + b;
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    if (!(threadIdx.x & 4)) r1[(size_t)s.b * 64 + half_parent(h) + 16 * q] = t;
  }
}

// e and its halo, with the coarse correction of each cell's parent (e1) when CORR
template <bool CORR, class T>
__device__ __forceinline__ void half_field(const Half& s, int h, const T* e, const T* e1, T (&own)[4][2], HaloV<T>& hv) {
#pragma unroll
  for (int k = 0; k < 4; ++k) ld2(e + s.c + 64 * k, own[k]);
  auto par = [](int i) {
    const int o = i & 511;
    return (size_t)(i >> 9) * 64 + ((o & 7) >> 1) + 4 * (((o >> 3) & 7) >> 1) + 16 * (o >> 7);
  };
  half_halo(
      s, hv, [&](int i) { return CORR ? e[i] + e1[par(i)] : e[i]; },
      [&](int i, T* o) {
        ld2(e + i, o);
        if (CORR) {
          const T a = e1[par(i)];
          o[0] += a;
          o[1] += a;
        }
      });
  if (CORR) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const T a = e1[(size_t)s.b * 64 + half_parent(h) + 16 * q];
#pragma unroll
      for (int k = 2 * q; k < 2 * q + 2; ++k) {
        own[k][0] += a;
        own[k][1] += a;
      }
    }
  }
}

// A Jacobi sweep of weight om into out (k0_post); returns the lane's part of r.out
template <class T, class DI>
__device__ __forceinline__ double half_sweep(const Half& s, const uint32_t (&mk)[4], DI dinv, const Params& P, T om,
                                             const T (&own)[4][2], const HaloV<T>& hv, const double (&r)[4][2], T* out) {
  const T ih2[3] = {(T)P.ih2[0], (T)P.ih2[1], (T)P.ih2[2]};
  double rz = 0;
  T w[2] = {};
  auto put = [&](int k, int j) {
    if (j == 1) st2(out + s.c + 64 * k, w[0], w[1]);
  };
  if (half_full(mk)) {
    const T di = dinv((uint16_t)kFullPair);
    half_each(own, hv, [&](int k, int j, const T* nb) {
      const T me = half_apply<true>((uint16_t)0, own[k][j], nb, ih2);
      w[j] = own[k][j] + om * di * ((T)r[k][j] - me);
      rz += r[k][j] * (double)w[j];
      put(k, j);
    });
  } else {
    half_each(own, hv, [&](int k, int j, const T* nb) {
      const uint16_t m = half_mask(mk, k, j);
      const T me = half_apply<false>(m, own[k][j], nb, ih2);
      w[j] = 0;
      if (m & kDomainBit) {
        w[j] = own[k][j] + om * dinv(m) * ((T)r[k][j] - me);
        rz += r[k][j] * (double)w[j];
      }
      put(k, j);
    });
  }
  return rz;
}

// p = z + beta p_old (first: z) on the half and its halo
template <class Z>
__device__ __forceinline__ void half_direction(const Half& s, const Z* z, const double* pold, double be, int first,
                                               double (&own)[4][2], HaloV<double>& hv) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    Z a[2];
    double b[2] = {0.0, 0.0};
    ld2(z + s.c + 64 * k, a);
    if (!first) ld2(pold + s.c + 64 * k, b);
#pragma unroll
    for (int j = 0; j < 2; ++j) own[k][j] = first ? (double)a[j] : (double)a[j] + be * b[j];
  }
  half_halo(
      s, hv, [&](int i) { return first ? (double)z[i] : (double)z[i] + be * pold[i]; },
      [&](int i, double* o) {
        Z a[2];
        double b[2] = {0.0, 0.0};
        ld2(z + i, a);
        if (!first) ld2(pold + i, b);
#pragma unroll
        for (int j = 0; j < 2; ++j) o[j] = first ? (double)a[j] : (double)a[j] + be * b[j];
      });
}

// q = M p (k_update_spmv); returns the lane's part of p.q
__device__ __forceinline__ double half_spmv(const Half& s, const uint32_t (&mk)[4], const Params& P, const double (&own)[4][2],
                                            const HaloV<double>& hv, double* pnew, double* q) {
  double pq = 0, w[2] = {};
  if (half_full(mk)) {
    half_each(own, hv, [&](int k, int j, const double* nb) {
      w[j] = half_apply<true>((uint16_t)0, own[k][j], nb, P.ih2);
      pq += own[k][j] * w[j];
      if (j == 1) {
        st2(q + s.c + 64 * k, w[0], w[1]);
        st2(pnew + s.c + 64 * k, own[k][0], own[k][1]);
      }
    });
  } else {
    double pc[2] = {};
    half_each(own, hv, [&](int k, int j, const double* nb) {
      const uint16_t m = half_mask(mk, k, j);
      const bool in = m & kDomainBit;
      const double a = half_apply<false>(m, own[k][j], nb, P.ih2);
      w[j] = in ? a : 0.0;
      pc[j] = in ? own[k][j] : 0.0;
      if (in) pq += own[k][j] * a;
      if (j == 1) {
        st2(q + s.c + 64 * k, w[0], w[1]);
        st2(pnew + s.c + 64 * k, pc[0], pc[1]);
      }
    });
  }
  return pq;
}

}  // namespace mac

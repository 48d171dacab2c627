// film_any.cuh -- Douglas ADI sweeps (Film_CK_AD/Film_3D/Geometry_Modules/
// mod_realspace.f90:22-140) on lines of any length, in FP32 and FP64.
//
// Delta form.  With M_x, M_y, M_z the implicit parts of the three sweeps
// (M_z with the field term ds w / 2), the step
//   (1 + M_x) q*  = [1 - M_x - 2 M_y - 2 M_z] q
//   (1 + M_y) q** = q* + M_y q
//   (1 + M_z) q'  = q** + M_z q
// is (1 + M_x) d1 = -2 (M_x + M_y + M_z) q, (1 + M_y) d2 = d1, (1 + M_z) d3 =
// d2, q' = q + d3 (walls d3 = -q): the y and z sweeps have no right-hand side
// to form and the intermediate arrays hold increments of O(ds).
//
// Lines are solved by G lanes with K or K - 1 rows each (fw::solve, n = gx,
// gy or gz + 1 rows dealt as evenly as they go, K = ceil(n / G) in 3..5), so
// a line length needs no factor:
//   k_adi_xy_any: one block per interior plane and chain; the plane of q and
//     the increments stay in shared memory through both sweeps;
//   k_adi_z_any: one block per tile of neighbouring lines and chain, staged
//     through shared memory (coalesced rows).
// z lines whose systems are not diagonally dominant (ds w / 2 below -0.99)
// run the reference's serial recurrence, with its pivots and their checks.
//
// The x and y matrices are the same for every line of a sweep: their factors
// are made once a propagation and applied line after line.
//
// Two planes have to fit a block's shared memory: in FP64 up to 120 x 120 points.
//
// Bound: FP64 the FP64 pipe and a last wave of planes (two chains of gz - 1 on 152
// SMs) that is not full, FP32 latency.
// A step of both chains, thread per line -> here: 20x35x100 FP64 220 -> 40 us
// (53 with factors made by every warp, 69 line by line), FP32 43.5 -> 12.5;
// 48^3 FP64 49 us, FP32 69.5 -> 11.9; 96x96x64 FP32 175 -> 25.
#pragma once
#include "film_warp.cuh"

namespace adiany {

// G of a line of n rows: K = ceil(n / G) in 3..5 and no lane of less than two
// rows; 0: none
__host__ __device__ inline int lanes(int n) {
  return n < 9 || n > 160 ? 0 : n <= 20 ? 4 : n <= 40 ? 8 : n <= 80 ? 16 : 32;
}

struct Rows {
  int start, i0;   // entry i >= i0 is row start + i - i0
};
template <int G, int K>
__device__ __forceinline__ Rows rows_of(int n, int gl) {
  const int base = n / G, extra = n - base * G;
  const int m = base + (gl < extra ? 1 : 0);
  return Rows{gl * base + min(gl, extra), K - m};
}

template <typename T>
struct Coef {
  T ax, ay, ds, hds;
};
template <typename T>
__device__ __forceinline__ Coef<T> coef(const FilmDev<T>& F, int dir, int s) {
  if constexpr (sizeof(T) == 4) {
    const AdiCoef c = adi_coef(F, dir, s);
    return Coef<T>{c.ax, c.ay, c.dsf, c.hdsf};
  } else {
    const double ds = film_ds(F.dss, dir, s, F.ns);
    return Coef<T>{-ds * F.hx2, -ds * F.hy2, ds, 0.5 * ds};
  }
}
template <typename T>
__device__ __forceinline__ T mesh(const FilmDev<T>& F, int j, int which) {   // 0 alpha, 1 gamma, 2 beta
  if constexpr (sizeof(T) == 4) return which == 0 ? F.alf[j] : which == 1 ? F.gaf[j] : F.bef[j];
  else return which == 0 ? F.alpha[j] : which == 1 ? F.gamma[j] : F.beta[j];
}
// the step's field
template <typename T>
__device__ __forceinline__ T fieldv(const FilmDev<T>& F, const double* w, int ty, size_t i) {
  if constexpr (sizeof(T) == 4) return __ldg(F.wf + (size_t)ty * F.npts + i);
  else return __ldg(w + (size_t)ty * F.npts + i);
}

// 2 M q of one axis from the differences to the two neighbours
template <typename T>
__device__ __forceinline__ T pair(T a, T c, T qm, T q0, T qp) {
  return r_fma(a, r_sub(qm, q0), r_mul(c, r_sub(qp, q0)));
}

// Factors of the periodic matrix (a, d, a) of the x and y lines, the same for
// every line and plane of a step: made once a propagation for every schedule
// entry (k_adi_any_factors), applied line after line (solve: fw::solve's
// operations on the right-hand side alone, about 5 a row where the whole
// solve takes 30).  Stored by value, then lane of the line.
constexpr int kFacVals = 5 * 4 + 2 * 5 + 1;   // K = 5, 32 lanes
constexpr int kFacAxis = kFacVals * 32;
template <typename T, int G, int K>
struct Factors {
  static constexpr int LG = G == 4 ? 2 : G == 8 ? 3 : G == 16 ? 4 : 5;
  T bet[K - 1], m[K - 1], g[K - 1], y[K - 1], z[K - 1];
  T kl[LG], kr[LG], iden, a;
  int i0;

  __device__ __forceinline__ Factors(T a_, T d_, int i0_, int* err) : a(a_), i0(i0_) {
    const unsigned mask = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), base = lane - gl;
    T b = (T)1;
#pragma unroll
    for (int i = 0; i < K - 1; ++i) {
      const bool pad = i < i0;
      const T ai = pad ? (T)-1 : a, di = pad ? (T)1 : d_;
      const T cm = i > 0 && !(i - 1 < i0) ? a : (T)0;       // super-diagonal of the row above
      g[i] = i == 0 ? (T)0 : r_mul(cm, b);
      const T piv = i == 0 ? di : r_fma(-ai, g[i], di);
      if (piv == (T)0) atomicOr(err, 1);
      b = fw::rcp(piv);
      bet[i] = b;
      m[i] = r_mul(-ai, b);
      y[i] = i == 0 ? m[0] : r_mul(m[i], y[i > 0 ? i - 1 : 0]);
      z[i] = i == K - 2 ? r_mul(-a, b) : (T)0;
    }
#pragma unroll
    for (int i = K - 3; i >= 0; --i) {
      y[i] = r_fma(-g[i + 1], y[i + 1], y[i]);
      z[i] = r_mul(-g[i + 1], z[i + 1]);
    }
    const int nx = base + ((gl + 1) & (G - 1));
    const T yn = __shfl_sync(mask, i0 ? y[1] : y[0], nx), zn = __shfl_sync(mask, i0 ? z[1] : z[0], nx);
    T A = r_mul(a, y[K - 2]), B = r_fma(a, yn, r_fma(a, z[K - 2], d_)), C = r_mul(a, zn);
#pragma unroll
    for (int s = 0; s < LG; ++s) {
      const int st = 1 << s, su = base + ((gl - st) & (G - 1)), sd = base + ((gl + st) & (G - 1));
      if (B == (T)0) atomicOr(err, 1);
      const T i1 = fw::rcp(B);
      kl[s] = r_mul(A, __shfl_sync(mask, i1, su));
      kr[s] = r_mul(C, __shfl_sync(mask, i1, sd));
      const T Au = __shfl_sync(mask, A, su), Cu = __shfl_sync(mask, C, su);
      const T Ad = __shfl_sync(mask, A, sd), Cd = __shfl_sync(mask, C, sd);
      B = r_fma(-kr[s], Ad, r_fma(-kl[s], Cu, B));
      A = r_mul(-kl[s], Au);
      C = r_mul(-kr[s], Cd);
    }
    const T den = r_add(r_add(A, C), B);
    if (den == (T)0) atomicOr(err, 1);
    iden = fw::rcp(den);
  }

  template <typename Op>
  __device__ __forceinline__ void each(Op op) {
    int k = 0;
#pragma unroll
    for (int i = 0; i < K - 1; ++i) {
      op(bet[i], k++); op(m[i], k++); op(g[i], k++); op(y[i], k++); op(z[i], k++);
    }
#pragma unroll
    for (int i = 0; i < LG; ++i) { op(kl[i], k++); op(kr[i], k++); }
    op(iden, k);
  }
  __device__ __forceinline__ void store(T* tab, int gl) {
    each([&](T v, int k) { tab[k * G + gl] = v; });
  }
  __device__ __forceinline__ Factors(T a_, int i0_, const T* tab, int gl) : a(a_), i0(i0_) {
    each([&](T& v, int k) { v = __ldg(tab + k * G + gl); });
  }

  // r: right-hand side of the lane's entries (0 in a pad entry); the solution
  // on return
  __device__ __forceinline__ void solve(T (&r)[K]) const {
    const unsigned mask = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), base = lane - gl;
    T x[K - 1];
#pragma unroll
    for (int i = 0; i < K - 1; ++i)
      x[i] = i == 0 ? r_mul(r[0], bet[0]) : r_fma(m[i], x[i > 0 ? i - 1 : 0], r_mul(r[i], bet[i]));
#pragma unroll
    for (int i = K - 3; i >= 0; --i) x[i] = r_fma(-g[i + 1], x[i + 1], x[i]);
    const T xn = __shfl_sync(mask, i0 ? x[1] : x[0], base + ((gl + 1) & (G - 1)));
    T R = r_fma(-a, xn, r_fma(-a, x[K - 2], r[K - 1]));
#pragma unroll
    for (int s = 0; s < LG; ++s) {
      const int st = 1 << s;
      const T Ru = __shfl_sync(mask, R, base + ((gl - st) & (G - 1)));
      const T Rd = __shfl_sync(mask, R, base + ((gl + st) & (G - 1)));
      R = r_fma(-kr[s], Rd, r_fma(-kl[s], Ru, R));
    }
    const T v = r_mul(R, iden);
    const T vl = __shfl_sync(mask, v, base + ((gl - 1) & (G - 1)));
#pragma unroll
    for (int i = 0; i < K - 1; ++i) r[i] = r_fma(z[i], v, r_fma(y[i], vl, x[i]));
    r[K - 1] = v;
  }
};

// x sweep of the plane P ([y][x], pitch pt) into D
template <typename T, int G, int K>
__device__ __forceinline__ void x_lines(const FilmDev<T>& F, const Coef<T>& cf, const T* P, T* D, int pt, const T* p0,
                                        const double* w, int ty, int z, const T* tab) {
  const int gx = F.gx, gy = F.gy, L = F.nlines;
  const int gl = threadIdx.x & (G - 1), ng = blockDim.x / G;
  const Rows R = rows_of<G, K>(gx, gl);
  const T az = r_mul(-cf.ds, mesh(F, z, 0)), cz = r_mul(-cf.ds, mesh(F, z, 1));
  const Factors<T, G, K> fac(cf.ax, R.i0, tab, gl);
  // a warp leaves when its lines are done (its lanes stay together)
  for (int y0 = (threadIdx.x & ~31) / G; y0 < gy; y0 += ng) {
    const int yl = y0 + (threadIdx.x & 31) / G;
    const bool live = yl < gy;
    const int y = live ? yl : 0;
    const int ym = (y == 0 ? gy : y) - 1, yp = y == gy - 1 ? 0 : y + 1;
    T r[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      r[i] = (T)0;
      if (i >= R.i0) {
        const int x = R.start + i - R.i0;
        const int xm = (x == 0 ? gx : x) - 1, xp = x == gx - 1 ? 0 : x + 1;
        const size_t g = (size_t)z * L + (size_t)y * gx + x;
        const T q0 = P[y * pt + x];
        T t = pair(cf.ax, cf.ax, P[y * pt + xm], q0, P[y * pt + xp]);
        t = r_add(t, pair(cf.ay, cf.ay, P[ym * pt + x], q0, P[yp * pt + x]));
        t = r_add(t, pair(az, cz, __ldg(p0 + g - L), q0, __ldg(p0 + g + L)));
        t = r_fma(r_mul(cf.hds, fieldv(F, w, ty, g)), q0, t);
        r[i] = r_mul((T)-2, t);
      }
    }
    fac.solve(r);
    if (live) {
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i >= R.i0) D[y * pt + R.start + i - R.i0] = r[i];
    }
  }
}

// y sweep of the increments D in place
template <typename T, int G, int K>
__device__ __forceinline__ void y_lines(const FilmDev<T>& F, const Coef<T>& cf, T* D, int pt, const T* tab) {
  const int gx = F.gx, gy = F.gy;
  const int gl = threadIdx.x & (G - 1), ng = blockDim.x / G;
  const Rows R = rows_of<G, K>(gy, gl);
  const Factors<T, G, K> fac(cf.ay, R.i0, tab, gl);
  for (int x0 = (threadIdx.x & ~31) / G; x0 < gx; x0 += ng) {
    const int xl = x0 + (threadIdx.x & 31) / G;
    const bool live = xl < gx;
    const int x = live ? xl : 0;
    T r[K];
#pragma unroll
    for (int i = 0; i < K; ++i) r[i] = i >= R.i0 ? D[(R.start + i - R.i0) * pt + x] : (T)0;
    fac.solve(r);
    if (live) {
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (i >= R.i0) D[(R.start + i - R.i0) * pt + x] = r[i];
    }
  }
}

// whether ds w / 2 < -0.99 (FP64 compares run on the narrow pipe: the high
// words order negative numbers by magnitude)
__device__ __forceinline__ bool far_below(float hw) { return hw < -0.99f; }
__device__ __forceinline__ bool far_below(double hw) {
  return (unsigned)__double2hiint(hw) >= 0xBFEFAE14u;   // -0.99 and below (and NaN of that sign)
}

// z sweep of a tile: D increments (the result in place), W field, [row][line]
// at pitch pt; tab: alpha, gamma, beta; lines [0, cnt) of the tile exist
template <typename T, int G, int K>
__device__ __forceinline__ void z_lines(const FilmDev<T>& F, const Coef<T>& cf, T* D, T* W, const T* tab, int pt,
                                        int cnt, int* dummy) {
  const int n = F.gz + 1;
  const int gl = threadIdx.x & (G - 1), ng = blockDim.x / G;
  const Rows R = rows_of<G, K>(n, gl);
  const T *al = tab, *ga = tab + n, *be = tab + 2 * n;
  for (int l0 = (threadIdx.x & ~31) / G; l0 < cnt; l0 += ng) {
    const int ll = l0 + (threadIdx.x & 31) / G;
    const bool live = ll < cnt;
    const int l = live ? ll : 0;
    T a[K], d[K], c[K], r[K];
    bool low = false;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      a[i] = (T)-1; d[i] = (T)1; c[i] = (T)0; r[i] = (T)0;
      if (i >= R.i0) {
        const int j = R.start + i - R.i0;
        r[i] = D[j * pt + l];
        if (j == 0 || j == n - 1) {
          a[i] = (T)0;
        } else {
          const T hw = r_mul(cf.hds, W[j * pt + l]);
          low |= far_below(hw);
          a[i] = r_mul(-cf.ds, al[j]);
          c[i] = r_mul(-cf.ds, ga[j]);
          d[i] = r_add(r_fma(cf.ds, be[j], (T)1), hw);
        }
      }
    }
    const unsigned any = __ballot_sync(0xffffffffu, low);
    const unsigned mine = (G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    const bool serial = (any & mine) != 0;
    fw::solve<G, K>(a, d, c, r, false, serial ? dummy : F.err, R.i0);
    if (!serial) {
      if (live) {
#pragma unroll
        for (int i = 0; i < K; ++i)
          if (i >= R.i0) D[(R.start + i - R.i0) * pt + l] = r[i];
      }
    } else if (live && gl == 0) {
      T bet = (T)1, cprev = (T)0, u = D[l];
      for (int j = 1; j < n; ++j) {
        T aj = (T)0, cj = (T)0, dj = (T)1;
        if (j < n - 1) {
          aj = r_mul(-cf.ds, al[j]);
          cj = r_mul(-cf.ds, ga[j]);
          dj = r_add(r_fma(cf.ds, be[j], (T)1), r_mul(cf.hds, W[j * pt + l]));
        }
        W[j * pt + l] = thomas_row<T>(bet, cprev, u, aj, cj, dj, D[j * pt + l], F.err);
        D[j * pt + l] = u;
      }
      for (int j = n - 2; j >= 0; --j) {
        u = r_fma(-W[(j + 1) * pt + l], u, D[j * pt + l]);
        D[j * pt + l] = u;
      }
    }
    __syncwarp();
  }
}

#define ADSCF_ANY_SHAPE(n, CALL)                               \
  switch (adiany::lanes(n) * 8 + ((n) + adiany::lanes(n) - 1) / adiany::lanes(n)) { \
    case 4 * 8 + 3: CALL(4, 3); break;                         \
    case 4 * 8 + 4: CALL(4, 4); break;                         \
    case 4 * 8 + 5: CALL(4, 5); break;                         \
    case 8 * 8 + 3: CALL(8, 3); break;                         \
    case 8 * 8 + 4: CALL(8, 4); break;                         \
    case 8 * 8 + 5: CALL(8, 5); break;                         \
    case 16 * 8 + 3: CALL(16, 3); break;                       \
    case 16 * 8 + 4: CALL(16, 4); break;                       \
    case 16 * 8 + 5: CALL(16, 5); break;                       \
    case 32 * 8 + 3: CALL(32, 3); break;                       \
    case 32 * 8 + 4: CALL(32, 4); break;                       \
    default: CALL(32, 5); break;                               \
  }

}  // namespace adiany

// Factors of schedule entry 1 + blockIdx.x: x lines by warp 0, y lines by warp 1
template <typename T>
__global__ void __launch_bounds__(64)
k_adi_any_factors(FilmDev<T> F) {
  const int k = 1 + blockIdx.x, lane = threadIdx.x & 31;
  const adiany::Coef<T> cf = adiany::coef(F, 0, k);
  T* tab = F.fac + (size_t)k * (2 * adiany::kFacAxis);
  const bool x = threadIdx.x < 32;
  const T a = x ? cf.ax : cf.ay, d = r_fma((T)-2, a, (T)1);
  const int n = x ? F.gx : F.gy;
  if (!x) tab += adiany::kFacAxis;
#define ADSCF_ANY_CALL(G, K)                                                                        \
  {                                                                                                 \
    adiany::Factors<T, G, K> f(a, d, adiany::rows_of<G, K>(n, lane & (G - 1)).i0, F.err);           \
    if (lane < G) f.store(tab, lane);                                                               \
  }
  ADSCF_ANY_SHAPE(n, ADSCF_ANY_CALL)
#undef ADSCF_ANY_CALL
}

// x and y sweeps of interior plane 1 + blockIdx.x, chain blockIdx.y.  Shared
// memory: two planes of gy rows at pitch gx | 1.
template <typename T>
__global__ void __launch_bounds__(512)
k_adi_xy_any(FilmDev<T> F, FieldRef fr, int s) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int gx = F.gx, gy = F.gy, L = F.nlines, pt = gx | 1;
  T* P = reinterpret_cast<T*>(smraw);
  T* D = P + (size_t)gy * pt;
  const int z = 1 + blockIdx.x, dir = blockIdx.y;
  const adiany::Coef<T> cf = adiany::coef(F, dir, s);
  const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
  const double* w = sizeof(T) == 4 ? nullptr : fr.get();
  const T* tab = F.fac + (size_t)(dir == 0 ? s : F.ns + 1 - s) * (2 * adiany::kFacAxis);
  const T* p0 = (dir == 0 ? F.q : F.qd) + (size_t)(s - 1) * F.npts;
  T* out = F.w1 + (size_t)dir * F.npts + (size_t)z * L;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int y = threadIdx.x >> 5; y < gy; y += nw)
    for (int x = lane; x < gx; x += 32) P[y * pt + x] = __ldg(p0 + (size_t)z * L + (size_t)y * gx + x);
  __syncthreads();
#define ADSCF_ANY_CALL(G, K) adiany::x_lines<T, G, K>(F, cf, P, D, pt, p0, w, ty, z, tab)
  ADSCF_ANY_SHAPE(gx, ADSCF_ANY_CALL)
#undef ADSCF_ANY_CALL
  __syncthreads();
#define ADSCF_ANY_CALL(G, K) adiany::y_lines<T, G, K>(F, cf, D, pt, tab + adiany::kFacAxis)
  ADSCF_ANY_SHAPE(gy, ADSCF_ANY_CALL)
#undef ADSCF_ANY_CALL
  __syncthreads();
  for (int y = threadIdx.x >> 5; y < gy; y += nw)
    for (int x = lane; x < gx; x += 32) out[(size_t)y * gx + x] = D[y * pt + x];
}

// z sweep of lines [blockIdx.x tl, + tl) of chain blockIdx.y (tl a power of
// two, at most 32).  Shared memory: increments and field, n rows at pitch tl
// + 1, three mesh tables, and a word for the pivot flags of solves that the
// serial recurrence replaces.
template <typename T>
__global__ void __launch_bounds__(512)
k_adi_z_any(FilmDev<T> F, FieldRef fr, int s, int tl) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = F.gz + 1, L = F.nlines, pt = tl + 1;
  T* D = reinterpret_cast<T*>(smraw);
  T* W = D + (size_t)n * pt;
  T* tab = W + (size_t)n * pt;
  int* dummy = reinterpret_cast<int*>(tab + 3 * n);
  const int l0 = blockIdx.x * tl, cnt = min(tl, L - l0), dir = blockIdx.y;
  const adiany::Coef<T> cf = adiany::coef(F, dir, s);
  const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
  const double* w = sizeof(T) == 4 ? nullptr : fr.get();
  const T* p0 = (dir == 0 ? F.q : F.qd) + (size_t)(s - 1) * F.npts;
  const T* w1 = F.w1 + (size_t)dir * F.npts;
  T* qn = (dir == 0 ? F.q : F.qd) + (size_t)s * F.npts;
  for (int i = threadIdx.x; i < 3 * n; i += blockDim.x) tab[i] = adiany::mesh(F, i % n, i / n);
  const int lx = threadIdx.x & (tl - 1), rj = threadIdx.x / tl, nr = blockDim.x / tl;
  for (int j = rj; j < n; j += nr) {
    T d = (T)0, v = (T)0;
    if (lx < cnt) {
      const size_t g = (size_t)j * L + l0 + lx;
      if (j == 0 || j == n - 1) {
        d = -__ldg(p0 + g);
      } else {
        d = __ldg(w1 + g);
        v = adiany::fieldv(F, w, ty, g);
      }
    }
    D[j * pt + lx] = d;
    W[j * pt + lx] = v;
  }
  __syncthreads();
#define ADSCF_ANY_CALL(G, K) adiany::z_lines<T, G, K>(F, cf, D, W, tab, pt, cnt, dummy)
  ADSCF_ANY_SHAPE(n, ADSCF_ANY_CALL)
#undef ADSCF_ANY_CALL
  __syncthreads();
  for (int j = rj; j < n; j += nr) {
    if (lx >= cnt) continue;
    const size_t g = (size_t)j * L + l0 + lx;
    const bool wall = j == 0 || j == n - 1;
    qn[g] = wall ? (T)0 : r_add(__ldg(p0 + g), D[j * pt + lx]);
  }
}

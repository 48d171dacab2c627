// film_line.cuh -- FP64 Crank-Nicolson chains of one-line films and brushes of up
// to 1024 rows (the systems of film_warp.cuh: (1 + ds M) u = q, q' = 2 u - q).
//
// The matrices of a contour depend on the field and the step alone, not on the
// propagator, and both chains meet the same ones.  A solve is therefore written
// as factors (make_factors) and their use (apply_factors): 5 FP64 operations a
// row and some 20 a lane, where elimination takes 16 and 90.  Two ways of
// running it do the same operations on the same numbers, so that their results
// are the same bits:
//   k_line_factors, k_line_chain: the factors of all ns steps at once on all SMs,
//     then a block per chain that only applies them;
//   k_line_elim, k_line_elim_b: a chain makes each step's factors as it goes
//     (batches, contexts of more lines than find an SM each, single steps, and
//     wherever the factors have no memory).
//
// Rows: one warp of K = 2..8 rows a lane up to 256 rows, four warps (one per
// quarter of an SM) beyond, K = 3..8.  The partition is film1d_chain_group's:
// interior rows in the left and own separator, the warp's separators by cyclic
// reduction, with four warps the warp's two boundary unknowns as further
// right-hand sides and the four warps' last rows by cyclic reduction again (one
// barrier a step).  What a thread needs of a step made ahead lies as kPairs
// double2 at stride of the line's threads, so it copies its own ahead of use
// (cp.async, two steps ahead) and meets no bank conflict.
//
// Bound: FP64 issue (64 to 76 cycles a warp instruction, 5 K + 17 of them a step
// with one warp, 5 K + 22 with four), then 11 to 12 shuffles and a barrier.
#pragma once
#include "film_warp.cuh"

namespace fl {

constexpr int kThreads = 128, kStages = 4, kMaxK = 8, kMaxRows = kThreads * kMaxK;
__host__ __device__ constexpr int warps_per_line(int n) { return n <= kFilmWarpRows ? 1 : 4; }
__host__ __device__ constexpr int rows_per_lane(int n) {
  return n <= 64 ? 2 : n <= kFilmWarpRows ? (n + 31) / 32 : (n + 127) / 128;
}

// slots of a thread's factors: reciprocal pivots, sub-diagonals times them,
// super-diagonals times the pivot above, responses to the left (y) and own (z)
// separator, the separator's row, reduction factors, then the warps' system
template <int K, int W>
struct Slot {
  static constexpr int bet = 0, m = bet + K - 1, g = m + K - 2, y = g + K - 2, z = y + K - 1;   // m, g from row 1
  static constexpr int aS = z + K - 1, cS = aS + 1, kl = cS + 1, kr = kl + 5, iB = kr + 5;
  static constexpr int As = iB + 1, Y = As + 1, Z = Y + 1, cc = Z + 1, kl2 = cc + 1, kr2 = kl2 + 2, iB2 = kr2 + 2;
  static constexpr int n = W == 1 ? iB + 1 : iB2 + 1, pairs = (n + 1) / 2;
};
inline size_t step_bytes(int rows) {
  const int K = rows_per_lane(rows), W = warps_per_line(rows);
  return (size_t)((5 * K + (W == 1 ? 6 : 15) + 1) / 2) * 32 * W * sizeof(double2);
}

// shared numbers of the four warps of a line
struct Exchange {
  double row[5][4];             // factors: last row's equation, first row's responses
  double rhs[2][2][5];          // by step parity: last rows' right-hand sides, first rows (a zero behind them)
};

// A thread's rows of a step: matrix entries from the mesh factors al, ga and the
// step's term t = beta + w / 2 (identity on the walls and past the line's end)
template <int K, typename Mesh>
__device__ __forceinline__ void line_rows(int j0, int n, double ds, const Mesh& mesh, double (&a)[K], double (&d)[K],
                                          double (&c)[K]) {
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int j = j0 + i;
    a[i] = 0.0; d[i] = 1.0; c[i] = 0.0;
    if (j > 0 && j < n - 1) {
      double al, ga, t;
      mesh(i, j, al, ga, t);
      a[i] = r_mul(-ds, al);
      c[i] = r_mul(-ds, ga);
      d[i] = r_fma(ds, t, 1.0);
    }
  }
}

// Factors of one system.  Only diagonally dominant lines use them
// (film_line_dominant), whose pivots cannot vanish, so none are looked at.  W =
// 4: every thread of the line's block, one barrier.
template <int K, int W>
__device__ __forceinline__ void make_factors(const double (&a)[K], const double (&d)[K], const double (&c)[K],
                                             double (&v)[2 * Slot<K, W>::pairs], Exchange* ex) {
  using S = Slot<K, W>;
  constexpr int Sp = K - 1, Li = K - 2;
  const unsigned mask = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  double y[K - 1], z[K - 1], g[K - 1], bet = 1.0;
  v[2 * S::pairs - 1] = 0.0;
#pragma unroll
  for (int i = 0; i < K - 1; ++i) {
    const int im = i > 0 ? i - 1 : 0;
    g[i] = i == 0 ? 0.0 : r_mul(c[im], bet);
    bet = fw::rcp(i == 0 ? d[0] : r_fma(-a[i], g[i], d[i]));
    const double mi = r_mul(-a[i], bet);
    v[S::bet + i] = bet;
    if (i > 0) {
      v[S::m + i - 1] = mi;
      v[S::g + i - 1] = g[i];
    }
    y[i] = i == 0 ? mi : r_mul(mi, y[im]);
    z[i] = i == Li ? r_mul(-c[i], bet) : 0.0;
  }
#pragma unroll
  for (int i = K - 3; i >= 0; --i) {
    y[i] = r_fma(-g[i + 1], y[i + 1], y[i]);
    z[i] = r_mul(-g[i + 1], z[i + 1]);
  }
#pragma unroll
  for (int i = 0; i < K - 1; ++i) {
    v[S::y + i] = y[i];
    v[S::z + i] = z[i];
  }
  const double yn = __shfl_down_sync(mask, y[0], 1), zn = __shfl_down_sync(mask, z[0], 1);
  const double As = r_mul(a[Sp], y[Li]), Bs = r_fma(a[Sp], z[Li], d[Sp]);
  v[S::aS] = a[Sp];
  v[S::cS] = c[Sp];
  // one warp: row 0 and the last row couple to nothing outside, and lane 31's
  // separator is that last row or past it, so the wrapped values below meet zeros
  double A = As, B = r_fma(c[Sp], yn, Bs), C = r_mul(c[Sp], zn), Y = 0.0, Z = 0.0;
  if constexpr (W > 1) {
    if (lane == 0) { Y = -A; A = 0.0; }
    if (lane == 30) { Z = -C; C = 0.0; }
    if (lane == 31) { A = 0.0; B = 1.0; C = 0.0; }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int su = (lane - (1 << k)) & 31, sd = (lane + (1 << k)) & 31;
    const double i0 = fw::rcp(B);
    const double kl = r_mul(A, __shfl_sync(mask, i0, su)), kr = r_mul(C, __shfl_sync(mask, i0, sd));
    v[S::kl + k] = kl;
    v[S::kr + k] = kr;
    const double Au = __shfl_sync(mask, A, su), Cu = __shfl_sync(mask, C, su);
    const double Ad = __shfl_sync(mask, A, sd), Cd = __shfl_sync(mask, C, sd);
    B = r_fma(-kr, Ad, r_fma(-kl, Cu, B));
    if constexpr (W > 1) {
      const double Yu = __shfl_sync(mask, Y, su), Zu = __shfl_sync(mask, Z, su);
      const double Yd = __shfl_sync(mask, Y, sd), Zd = __shfl_sync(mask, Z, sd);
      Y = r_fma(-kr, Yd, r_fma(-kl, Yu, Y));
      Z = r_fma(-kr, Zd, r_fma(-kl, Zu, Z));
    }
    A = r_mul(-kl, Au);
    C = r_mul(-kr, Cd);
  }
  double iB = fw::rcp(B);
  if constexpr (W == 1) {
    v[S::iB] = iB;
  } else {
    const int w = threadIdx.x >> 5;
    Y = r_mul(Y, iB);
    Z = r_mul(Z, iB);
    if (lane == 31) { iB = 0.0; Y = 0.0; Z = 1.0; }   // its separator is the warp's boundary unknown
    v[S::iB] = iB;
    v[S::As] = As;
    v[S::Y] = Y;
    v[S::Z] = Z;
    // the warp's last row in the boundary unknowns, and its first row
    const double Y30 = __shfl_up_sync(mask, Y, 1), Z30 = __shfl_up_sync(mask, Z, 1);
    if (lane == 31) {
      ex->row[0][w] = r_mul(As, Y30);
      ex->row[1][w] = r_fma(As, Z30, Bs);
      ex->row[2][w] = c[Sp];
    }
    if (lane == 0) {
      ex->row[3][w] = r_fma(z[0], Y, y[0]);
      ex->row[4][w] = r_mul(z[0], Z);
    }
    __syncthreads();
    // the warps' system, on every four lanes
    const int l = lane & 3, l4 = lane & ~3;
    const double cc = l + 1 < W ? ex->row[2][l] : 0.0;
    double gA = l > 0 ? ex->row[0][l] : 0.0, gB = ex->row[1][l], gC = 0.0;
    if (l + 1 < W) {
      gB = r_fma(cc, ex->row[3][l + 1], gB);
      gC = r_mul(cc, ex->row[4][l + 1]);
    }
    v[S::cc] = cc;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int su = l4 | ((l - (1 << k)) & 3), sd = l4 | ((l + (1 << k)) & 3);
      const double i0 = fw::rcp(gB);
      const double kl = r_mul(gA, __shfl_sync(mask, i0, su)), kr = r_mul(gC, __shfl_sync(mask, i0, sd));
      v[S::kl2 + k] = kl;
      v[S::kr2 + k] = kr;
      const double Au = __shfl_sync(mask, gA, su), Cu = __shfl_sync(mask, gC, su);
      const double Ad = __shfl_sync(mask, gA, sd), Cd = __shfl_sync(mask, gC, sd);
      gB = r_fma(-kr, Ad, r_fma(-kl, Cu, gB));
      gA = r_mul(-kl, Au);
      gC = r_mul(-kr, Cd);
    }
    v[S::iB2] = fw::rcp(gB);
  }
}

// q of the thread's rows j0.. to the next step: u solves with the factors f(slot);
// halve: the walls' q is not yet 0 (step 1).  `loaded` is called when the factors
// have been read but for those of the last rows.  W = 4: one barrier.
template <int K, int W, typename Get, typename Loaded>
__device__ __forceinline__ void apply_factors(double (&q)[K], int j0, int n, int s, bool halve, const Get& f, Exchange* ex,
                                              const Loaded& loaded) {
  using S = Slot<K, W>;
  constexpr int Sp = K - 1, Li = K - 2;
  const unsigned mask = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  double r[K], x[K - 1];
#pragma unroll
  for (int i = 0; i < K; ++i) r[i] = q[i];
  if (halve) {   // walls: u = q / 2, so q' = 0
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (j0 + i == 0 || j0 + i == n - 1) r[i] = r_mul(0.5, q[i]);
  }
  x[0] = r_mul(r[0], f(S::bet));
#pragma unroll
  for (int i = 1; i < K - 1; ++i) x[i] = r_fma(f(S::m + i - 1), x[i - 1], r_mul(r[i], f(S::bet + i)));
#pragma unroll
  for (int i = K - 3; i >= 0; --i) x[i] = r_fma(-f(S::g + i), x[i + 1], x[i]);
  const double xn = __shfl_down_sync(mask, x[0], 1);
  const double Rs = r_fma(-f(S::aS), x[Li], r[Sp]);
  double R = r_fma(-f(S::cS), xn, Rs);
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const double Ru = __shfl_sync(mask, R, (lane - (1 << k)) & 31), Rd = __shfl_sync(mask, R, (lane + (1 << k)) & 31);
    R = r_fma(-f(S::kr + k), Rd, r_fma(-f(S::kl + k), Ru, R));
  }
  const double X = r_mul(R, f(S::iB));
  double v = X, vl;
  if constexpr (W == 1) {
    vl = __shfl_up_sync(mask, v, 1);
    if (lane == 0) vl = 0.0;
  } else {
    const int w = threadIdx.x >> 5, l = lane & 3, l4 = lane & ~3;
    // lane 31: the right-hand side of the warp's last row; lane 0: its first row
    const double Xu = __shfl_up_sync(mask, X, 1);
    const bool last = lane == 31;
    const double e = r_fma(last ? -f(S::As) : f(S::z), last ? Xu : X, last ? Rs : x[0]);
    double (*E)[5] = ex->rhs[s & 1];
    if (last) E[0][w] = e;
    if (lane == 0) E[1][w] = e;
    __syncthreads();
    double G = r_fma(-f(S::cc), E[1][l + 1], E[0][l]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double Gu = __shfl_sync(mask, G, l4 | ((l - (1 << k)) & 3)), Gd = __shfl_sync(mask, G, l4 | ((l + (1 << k)) & 3));
      G = r_fma(-f(S::kr2 + k), Gd, r_fma(-f(S::kl2 + k), Gu, G));
    }
    const double U = r_mul(G, f(S::iB2));
    const double UR = __shfl_sync(mask, U, w);
    double UL = __shfl_sync(mask, U, w > 0 ? w - 1 : 0);
    if (w == 0) UL = 0.0;
    v = r_fma(f(S::Z), UR, r_fma(f(S::Y), UL, X));
    vl = __shfl_up_sync(mask, v, 1);
    if (lane == 0) vl = UL;
  }
  loaded();
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int ii = i < Sp ? i : 0;
    const double u = i == Sp ? v : r_fma(f(S::z + ii), v, r_fma(f(S::y + ii), vl, x[ii]));
    q[i] = r_fma(2.0, u, -q[i]);
  }
}

// node 0 of the thread's rows (a single step starts from the propagator in place)
template <int K>
__device__ __forceinline__ void start_rows(const FilmDev<double>& F, int dir, double* chain, int j0, double (&q)[K]) {
  const int n = F.gz + 1;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    q[i] = 0.0;
    if (j0 + i < n) {
      double* at = chain + (size_t)(j0 + i) * F.nlines;
      q[i] = F.single ? *at : dir == 1 && F.brush ? F.graft[j0 + i] : 1.0;
      if (!F.single) *at = q[i];
    }
  }
}
template <int K>
__device__ __forceinline__ void store_rows(const FilmDev<double>& F, double* slice, int j0, const double (&q)[K]) {
  const int n = F.gz + 1;
#pragma unroll
  for (int i = 0; i < K; ++i)
    if (j0 + i < n) slice[(size_t)(j0 + i) * F.nlines] = q[i];
}

#define ADSCF_LINE_SHAPE(n, CALL)                                     \
  switch (fl::warps_per_line(n) * 8 + fl::rows_per_lane(n) - 1) {     \
    case 8 + 1: CALL(2, 1); break;                                    \
    case 8 + 2: CALL(3, 1); break;                                    \
    case 8 + 3: CALL(4, 1); break;                                    \
    case 8 + 4: CALL(5, 1); break;                                    \
    case 8 + 5: CALL(6, 1); break;                                    \
    case 8 + 6: CALL(7, 1); break;                                    \
    case 8 + 7: CALL(8, 1); break;                                    \
    case 32 + 2: CALL(3, 4); break;                                   \
    case 32 + 3: CALL(4, 4); break;                                   \
    case 32 + 4: CALL(5, 4); break;                                   \
    case 32 + 5: CALL(6, 4); break;                                   \
    case 32 + 6: CALL(7, 4); break;                                   \
    default: CALL(8, 4); break;                                       \
  }

// One chain, factors made step by step, by the line's W warps.  sm: the line's
// mesh factors and terms, [alpha, gamma, beta + w / 2 of type 0, of type 1][i][thread].
template <int K, int W>
__device__ __forceinline__ void chain_elim(const FilmDev<double>& F, int dir, double* chain, const double* field, double* sm,
                                           Exchange* ex) {
  using S = Slot<K, W>;
  constexpr int T = 32 * W;
  const int n = F.gz + 1, L = F.nlines, t = threadIdx.x & (T - 1), j0 = t * K;
  const bool two = F.ntypes == 2 && !F.single;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int j = j0 + i;
    if (j >= n) continue;
    sm[(0 * K + i) * T + t] = F.alpha[j];
    sm[(1 * K + i) * T + t] = F.gamma[j];
    sm[(2 * K + i) * T + t] = r_fma(0.5, field[(size_t)j * L], F.beta[j]);
    if (two) sm[(3 * K + i) * T + t] = r_fma(0.5, field[F.npts + (size_t)j * L], F.beta[j]);
  }
  double q[K];
  start_rows<K>(F, dir, chain, j0, q);
  if constexpr (W > 1) {
    if (t < 4) ex->rhs[t & 1][t >> 1][4] = 0.0;
    __syncthreads();
  }
  for (int s = 1; s <= F.ns; ++s) {
    const int ty = F.brush || F.single ? 0 : film_type(dir, s, F.ns, F.na);
    const double* term = sm + (2 + ty) * K * T + t;
    double v[2 * S::pairs], a[K], d[K], c[K];
    line_rows<K>(j0, n, film_ds(F.dss, dir, s, F.ns),
                 [&](int i, int, double& al, double& ga, double& tt) {
                   al = sm[i * T + t];
                   ga = sm[(K + i) * T + t];
                   tt = term[i * T];
                 },
                 a, d, c);
    make_factors<K, W>(a, d, c, v, ex);
    apply_factors<K, W>(q, j0, n, s, s == 1, [&](int i) { return v[i]; }, ex, [] {});
    store_rows<K>(F, chain + (size_t)s * F.npts, j0, q);
  }
}
__host__ __device__ constexpr size_t elim_bytes(int K) { return (size_t)4 * K * kThreads * sizeof(double); }

}  // namespace fl

// Factors of all steps of lines blockIdx.y, to fac[line][step][pair][thread]: a
// block of four warps makes those of one step (W = 4) or of four (W = 1)
template <int K, int W>
__global__ void __launch_bounds__(fl::kThreads)
k_line_factors(FilmDev<double> F, FieldRef fr, double2* __restrict__ fac) {
  using S = fl::Slot<K, W>;
  constexpr int T = 32 * W;
  __shared__ fl::Exchange ex;
  const int n = F.gz + 1, L = F.nlines, line = blockIdx.y, t = threadIdx.x & (T - 1);
  const int step = blockIdx.x * (fl::kThreads / T) + threadIdx.x / T + 1;
  if (step > F.ns) return;   // a whole warp (W = 1); W = 4 has no such block
  const double ds = F.dss[step];
  const int ty = F.brush ? 0 : film_type(0, step, F.ns, F.na);
  const double* wf = fr.get() + (size_t)ty * F.npts + line;
  double v[2 * S::pairs], a[K], d[K], c[K];
  fl::line_rows<K>(t * K, n, ds,
                   [&](int, int j, double& al, double& ga, double& tt) {
                     al = F.alpha[j];
                     ga = F.gamma[j];
                     tt = r_fma(0.5, wf[(size_t)j * L], F.beta[j]);
                   },
                   a, d, c);
  fl::make_factors<K, W>(a, d, c, v, &ex);
  double2* out = fac + ((size_t)line * F.ns + step - 1) * (S::pairs * T) + t;
#pragma unroll
  for (int p = 0; p < S::pairs; ++p) out[p * T] = make_double2(v[2 * p], v[2 * p + 1]);
}

// Chain blockIdx.y of line blockIdx.x, factors made ahead.  Dynamic shared
// memory: kStages steps of factors.  501 rows, 8 iterations of 100 steps 7.2 ->
// 2.2 ms, 1001 rows and 1200 steps 11.1 -> 4.1 ms against factors in the chain.
template <int K, int W>
__global__ void __launch_bounds__(32 * W, 1)
k_line_chain(FilmDev<double> F, FieldRef fr, const double2* __restrict__ fac, int* __restrict__ serial) {
  using S = fl::Slot<K, W>;
  constexpr int T = 32 * W, P = S::pairs * T;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ fl::Exchange ex;
  const int n = F.gz + 1, L = F.nlines, ns = F.ns, line = blockIdx.x, dir = blockIdx.y;
  if (film_line_serial<double>(F, fr.get(), line, dir, threadIdx.x == 0, serial)) return;
  double2* ring = reinterpret_cast<double2*>(smraw) + threadIdx.x;
  const double2* src = fac + (size_t)line * ns * P + threadIdx.x;
  auto fetch = [&](int s) {
    if (s <= ns) {
      const double2* from = src + (size_t)(dir == 0 ? s - 1 : ns - s) * P;
      const unsigned to = (unsigned)__cvta_generic_to_shared(ring + (s & (fl::kStages - 1)) * P);
#pragma unroll
      for (int p = 0; p < S::pairs; ++p)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + p * T * 16), "l"(from + p * T) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(1);
  fetch(2);
  double* chain = (dir == 0 ? F.q : F.qd) + line;
  const int j0 = threadIdx.x * K;
  double q[K];
  fl::start_rows<K>(F, dir, chain, j0, q);
  if constexpr (W > 1) {
    if (threadIdx.x < 4) ex.rhs[threadIdx.x & 1][threadIdx.x >> 1][4] = 0.0;
    __syncthreads();
  }
  for (int s = 1; s <= ns; ++s) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    const double2* St = ring + (s & (fl::kStages - 1)) * P;
    // a thread reads what it copied itself, and step s + 2 fills the stage of
    // step s - 2; its copies go out once this step's loads have (at the top of
    // the step they held those up: 1001 rows 4.43 against 4.11 ms)
    fl::apply_factors<K, W>(q, j0, n, s, s == 1, [&](int i) { return (i & 1) ? St[(i >> 1) * T].y : St[(i >> 1) * T].x; },
                            &ex, [&] { fetch(s + 2); });
    fl::store_rows<K>(F, chain + (size_t)s * F.npts, j0, q);
  }
}

// Chain blockIdx.y of lines (128 / 32 W a block) of one context
template <int K, int W>
__global__ void __launch_bounds__(fl::kThreads)
k_line_elim(FilmDev<double> F, FieldRef fr, int* __restrict__ serial) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ fl::Exchange ex;
  constexpr int T = 32 * W;
  const int sub = threadIdx.x / T, line = blockIdx.x * (fl::kThreads / T) + sub, dir = blockIdx.y;
  if (line >= F.nlines) return;
  if (film_line_serial<double>(F, fr.get(), line, dir, (threadIdx.x & (T - 1)) == 0, serial)) return;
  fl::chain_elim<K, W>(F, dir, (dir == 0 ? F.q : F.qd) + line, fr.get() + line,
                       reinterpret_cast<double*>(smraw) + sub * 4 * K * T, &ex);
}
// (film << 1) | chain of a batch's films of W warps a line, K by film: one launch
// for all lengths, so that short lines and long ones run beside each other.  Where
// none has more than KMAX = 4 rows a lane, five blocks an SM in place of two: 2048
// films of 40 to 60 rows 31.0 -> 28.0 us a step of both chains (118 registers, and
// 96 with 96 bytes of spill; no such gain for eight rows: 2048 films of 180 to 250
// rows 61.9 with 188 registers, 62.3 with 128).
template <int W, int KMAX>
__global__ void __launch_bounds__(fl::kThreads, KMAX <= 4 ? 5 : 1)
k_line_elim_b(const FilmDev<double>* __restrict__ Fs, const ScfDev* __restrict__ Ss, const int* __restrict__ items, int nitems,
              int* __restrict__ serial) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ fl::Exchange ex;
  constexpr int T = 32 * W;
  const int sub = threadIdx.x / T, it = blockIdx.x * (fl::kThreads / T) + sub;
  if (it >= nitems) return;
  const int f = items[it] >> 1, dir = items[it] & 1;
  const FilmDev<double> F = Fs[f];
  const ScfDev& S = Ss[f];
  const double* field = S.hx + (size_t)((*S.iter) % S.slots) * ((size_t)S.ntypes * S.npts);
  if (film_line_serial<double>(F, field, 0, dir, (threadIdx.x & (T - 1)) == 0, serial + f)) return;
  double* chain = dir == 0 ? F.q : F.qd;
  double* sm = reinterpret_cast<double*>(smraw) + sub * 4 * KMAX * T;
  switch (fl::rows_per_lane(F.gz + 1)) {
    case 2: if constexpr (W == 1) fl::chain_elim<2, W>(F, dir, chain, field, sm, &ex); break;
    case 3: fl::chain_elim<3, W>(F, dir, chain, field, sm, &ex); break;
    case 4: fl::chain_elim<4, W>(F, dir, chain, field, sm, &ex); break;
    case 5: if constexpr (KMAX > 4) fl::chain_elim<5, W>(F, dir, chain, field, sm, &ex); break;
    case 6: if constexpr (KMAX > 4) fl::chain_elim<6, W>(F, dir, chain, field, sm, &ex); break;
    case 7: if constexpr (KMAX > 4) fl::chain_elim<7, W>(F, dir, chain, field, sm, &ex); break;
    default: if constexpr (KMAX > 4) fl::chain_elim<8, W>(F, dir, chain, field, sm, &ex); break;
  }
}

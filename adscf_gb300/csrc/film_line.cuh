// film_line.cuh -- FP64 Crank-Nicolson chains of one-line films and brushes
// with the factors of every step made ahead (the systems of film_warp.cuh:
// (1 + ds M) u = q, q' = 2 u - q).
//
// The matrices of a contour depend on the field and the step alone, not on the
// propagator, and both chains meet the same ones.  k_line_factors eliminates
// the systems of all ns steps at once, a block per (step, line), on all SMs;
// k_line_chain then walks a chain and only applies them: 5 FP64 operations a
// row and some 20 a lane, where eliminating in the chain takes 16 and 90.
//
// One block of four warps (one per quarter of an SM) solves a line of up to
// 1024 rows, K = 2..8 rows a lane.  The partition is film1d_chain_group's:
// interior rows in the left and own separator, the warp's separators by cyclic
// reduction with the warp's two boundary unknowns as further right-hand sides,
// the four warps' last rows by cyclic reduction again; one barrier a step.
// What a thread needs of a step lies as kPairs double2 at stride 128, so it
// copies its own ahead of use (cp.async, two steps ahead) and meets no bank
// conflict.
//
// Bound: FP64 issue (76 cycles a warp instruction with four warps on an SM, 5 K
// + 22 of them a step), then 12 shuffles and a barrier.  8 iterations of a
// 501-row film with 100 steps 7.2 -> 2.2 ms, a 1001-row brush with 1200 steps
// 11.1 -> 4.1 ms against elimination in the chain.
#pragma once
#include "film_warp.cuh"

namespace fl {

constexpr int kWarps = 4, kThreads = 32 * kWarps, kStages = 4, kMaxK = 8;
constexpr int kMaxRows = kThreads * kMaxK;
__host__ __device__ constexpr int rows_per_lane(int n) { return n <= 2 * kThreads ? 2 : (n + kThreads - 1) / kThreads; }

// slots of a thread's factors: reciprocal pivots, sub-diagonals times them,
// super-diagonals times the pivot above, responses to the left (y) and own (z)
// separator, the separator's row, reduction factors, then the warps' system
template <int K>
struct Slot {
  static constexpr int bet = 0, m = bet + K - 1, g = m + K - 2, y = g + K - 2, z = y + K - 1;   // m, g from row 1
  static constexpr int aS = z + K - 1, cS = aS + 1, As = cS + 1, kl = As + 1, kr = kl + 5;
  static constexpr int iB = kr + 5, Y = iB + 1, Z = Y + 1, cc = Z + 1, kl2 = cc + 1, kr2 = kl2 + 2, iB2 = kr2 + 2;
  static constexpr int n = iB2 + 1, pairs = (n + 1) / 2;
};
inline size_t step_bytes(int K) { return (size_t)(5 * K + 16) / 2 * kThreads * sizeof(double2); }

}  // namespace fl

// Factors of steps blockIdx.x + 1 of line blockIdx.y, to fac[line][step][pair]
// [thread].  Only diagonally dominant lines use them (film_line_dominant), whose
// pivots cannot vanish, so none are looked at.
template <int K>
__global__ void __launch_bounds__(fl::kThreads)
k_line_factors(FilmDev<double> F, FieldRef fr, double2* __restrict__ fac) {
  using S = fl::Slot<K>;
  __shared__ double ex[5][fl::kWarps];
  constexpr int Sp = K - 1, Li = K - 2;
  const unsigned mask = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = F.gz + 1, L = F.nlines, line = blockIdx.y, step = blockIdx.x + 1;
  const double ds = F.dss[step];
  const int ty = F.brush ? 0 : film_type(0, step, F.ns, F.na);
  const double* wf = fr.get() + (size_t)ty * F.npts + line;
  double v[2 * S::pairs];
  v[2 * S::pairs - 1] = 0.0;
  double a[K], d[K], c[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int j = threadIdx.x * K + i;
    a[i] = 0.0; d[i] = 1.0; c[i] = 0.0;
    if (j > 0 && j < n - 1) {
      a[i] = r_mul(-ds, F.alpha[j]);
      c[i] = r_mul(-ds, F.gamma[j]);
      d[i] = r_fma(ds, r_fma(0.5, wf[(size_t)j * L], F.beta[j]), 1.0);
    }
  }
  double y[K - 1], z[K - 1], g[K - 1], bet = 1.0;
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
  v[S::As] = As;
  double A = As, B = r_fma(c[Sp], yn, Bs), C = r_mul(c[Sp], zn), Y = 0.0, Z = 0.0;
  if (lane == 0) { Y = -A; A = 0.0; }
  if (lane == 30) { Z = -C; C = 0.0; }
  if (lane == 31) { A = 0.0; B = 1.0; C = 0.0; }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int su = (lane - (1 << k)) & 31, sd = (lane + (1 << k)) & 31;
    const double i0 = fw::rcp(B);
    const double kl = r_mul(A, __shfl_sync(mask, i0, su)), kr = r_mul(C, __shfl_sync(mask, i0, sd));
    v[S::kl + k] = kl;
    v[S::kr + k] = kr;
    const double Au = __shfl_sync(mask, A, su), Cu = __shfl_sync(mask, C, su);
    const double Yu = __shfl_sync(mask, Y, su), Zu = __shfl_sync(mask, Z, su);
    const double Ad = __shfl_sync(mask, A, sd), Cd = __shfl_sync(mask, C, sd);
    const double Yd = __shfl_sync(mask, Y, sd), Zd = __shfl_sync(mask, Z, sd);
    B = r_fma(-kr, Ad, r_fma(-kl, Cu, B));
    Y = r_fma(-kr, Yd, r_fma(-kl, Yu, Y));
    Z = r_fma(-kr, Zd, r_fma(-kl, Zu, Z));
    A = r_mul(-kl, Au);
    C = r_mul(-kr, Cd);
  }
  double iB = fw::rcp(B);
  Y = r_mul(Y, iB);
  Z = r_mul(Z, iB);
  if (lane == 31) { iB = 0.0; Y = 0.0; Z = 1.0; }   // its separator is the warp's boundary unknown
  v[S::iB] = iB;
  v[S::Y] = Y;
  v[S::Z] = Z;
  // the warp's last row in the boundary unknowns, and its first row
  const double Y30 = __shfl_up_sync(mask, Y, 1), Z30 = __shfl_up_sync(mask, Z, 1);
  if (lane == 31) {
    ex[0][w] = r_mul(As, Y30);
    ex[1][w] = r_fma(As, Z30, Bs);
    ex[2][w] = c[Sp];
  }
  if (lane == 0) {
    ex[3][w] = r_fma(z[0], Y, y[0]);
    ex[4][w] = r_mul(z[0], Z);
  }
  __syncthreads();
  // the warps' system, on every four lanes
  const int l = lane & 3, l4 = lane & ~3;
  const double cc = l + 1 < fl::kWarps ? ex[2][l] : 0.0;
  double gA = l > 0 ? ex[0][l] : 0.0, gB = ex[1][l], gC = 0.0;
  if (l + 1 < fl::kWarps) {
    gB = r_fma(cc, ex[3][l + 1], gB);
    gC = r_mul(cc, ex[4][l + 1]);
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
  double2* out = fac + ((size_t)line * F.ns + blockIdx.x) * (S::pairs * fl::kThreads) + threadIdx.x;
#pragma unroll
  for (int p = 0; p < S::pairs; ++p) out[p * fl::kThreads] = make_double2(v[2 * p], v[2 * p + 1]);
}

// Chain blockIdx.y of line blockIdx.x.  Dynamic shared memory: kStages steps
// of factors.
template <int K>
__global__ void __launch_bounds__(fl::kThreads)
k_line_chain(FilmDev<double> F, FieldRef fr, const double2* __restrict__ fac) {
  using S = fl::Slot<K>;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double ex[2][2][fl::kWarps + 1];   // by step parity: last rows' right-hand sides, first rows
  constexpr int Sp = K - 1, Li = K - 2;
  const unsigned mask = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = F.gz + 1, L = F.nlines, ns = F.ns, line = blockIdx.x, dir = blockIdx.y;
  if (!film_line_dominant<double>(F, fr.get() + line, L)) {
    if (threadIdx.x == 0) film1d_chain<double>(F, fr.get(), line, dir);
    return;
  }
  double2* ring = reinterpret_cast<double2*>(smraw) + threadIdx.x;
  const double2* src = fac + (size_t)line * ns * (S::pairs * fl::kThreads) + threadIdx.x;
  auto fetch = [&](int s) {
    if (s <= ns) {
      const double2* from = src + (size_t)(dir == 0 ? s - 1 : ns - s) * (S::pairs * fl::kThreads);
      const unsigned to = (unsigned)__cvta_generic_to_shared(ring + (s & (fl::kStages - 1)) * (S::pairs * fl::kThreads));
#pragma unroll
      for (int p = 0; p < S::pairs; ++p)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + p * fl::kThreads * 16),
                     "l"(from + p * fl::kThreads) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(1);
  fetch(2);
  double* chain = (dir == 0 ? F.q : F.qd) + line;
  const int j0 = threadIdx.x * K;
  double q[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    q[i] = 0.0;
    if (j0 + i < n) {
      q[i] = dir == 1 && F.brush ? F.graft[j0 + i] : 1.0;
      chain[(size_t)(j0 + i) * L] = q[i];
    }
  }
  if (threadIdx.x < 4) ex[threadIdx.x & 1][threadIdx.x >> 1][fl::kWarps] = 0.0;
  __syncthreads();
  const int l = lane & 3, l4 = lane & ~3;
  for (int s = 1; s <= ns; ++s) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    const double2* P = ring + (s & (fl::kStages - 1)) * (S::pairs * fl::kThreads);
    auto f = [&](int i) { return (i & 1) ? P[(i >> 1) * fl::kThreads].y : P[(i >> 1) * fl::kThreads].x; };
    double r[K], x[K - 1];
#pragma unroll
    for (int i = 0; i < K; ++i) r[i] = q[i];
    if (s == 1) {   // walls: u = q / 2, so q' = 0
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
    // lane 31: the right-hand side of the warp's last row; lane 0: its first row
    const double Xu = __shfl_up_sync(mask, X, 1);
    const bool last = lane == 31;
    const double e = r_fma(last ? -f(S::As) : f(S::z), last ? Xu : X, last ? Rs : x[0]);
    double (*E)[fl::kWarps + 1] = ex[s & 1];
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
    const double v = r_fma(f(S::Z), UR, r_fma(f(S::Y), UL, X));
    double vl = __shfl_up_sync(mask, v, 1);
    if (lane == 0) vl = UL;
    // the stage that step s + 2 fills was last read in step s - 2, on the other
    // side of a barrier; its copies go out once this step's loads have (at the
    // top of the step they held those up: 1001 rows 4.43 against 4.11 ms)
    fetch(s + 2);
    double* qn = chain + (size_t)s * F.npts;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int ii = i < Sp ? i : 0;
      const double u = i == Sp ? v : r_fma(f(S::z + ii), v, r_fma(f(S::y + ii), vl, x[ii]));
      q[i] = r_fma(2.0, u, -q[i]);
      if (j0 + i < n) qn[(size_t)(j0 + i) * L] = q[i];
    }
  }
}

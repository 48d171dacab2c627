// film_warp.cuh -- cooperative tridiagonal line solves for the Crank-Nicolson
// sweeps of films and brushes: a warp, part of one, or several warps per line.
//
// The reference solves every line with a serial Thomas recurrence (tridiag,
// Film_CK_AD/Film_3D/Geometry_Modules/mod_realspace.f90:184-215; the 1D CN
// step of Film_1D/.../mod_realspace.f90:24-79).  One thread per line leaves
// a GB300 with a few warps per SM, each waiting on a chain of dependent
// operations as long as the line.  Here G lanes of a warp share one line:
//
//  - lane l owns the contiguous rows [s_l, e_l] of the line (a chunk of at
//    most M rows, held in registers across all contour steps); the last row
//    e_l of each chunk is a separator;
//  - each lane eliminates its interior rows [s_l, e_l - 1] once with three
//    right-hand sides, so that every interior unknown is
//    u_i = x_i + y_i u(e_{l-1}) + z_i u(e_l)   (left and own separator);
//  - substituting these into the separator rows gives one tridiagonal
//    equation per lane in the separators alone,
//    A_l u(e_{l-1}) + B_l u(e_l) + C_l u(e_{l+1}) = R_l,
//    solved by parallel cyclic reduction across the G lanes (log2 G steps of
//    shuffles); a periodic line closes the reduced system cyclically;
//  - the interior unknowns then follow from their lane's two separators.
//
// The matrix is that of the reference; only the elimination order differs,
// so the result equals the serial solve up to rounding (the systems are
// diagonally dominant: 1 + hw > 0 beyond the off-diagonals).  Pivots are
// multiplied by their reciprocals (FP32: rcp.approx, as the serial FP32
// sweeps); a zero pivot sets the error flag like the serial solve.  The FP32
// sweeps solve for the increment u = q' - q of the step (see cn_rhs), so
// Dirichlet rows give u = -q.
#pragma once
#include "film_kernels.cuh"

namespace fw {

// Reciprocal pivots.  FP32: the hardware reciprocal (see rcp_hw).  FP64: the
// hardware's approximation y (about 20 bits) and two Newton-Raphson steps y +=
// y (1 - x y): four FP64 instructions (each 64 cycles on its SM quarter) and
// no branch for the range ends, which a pivot of 1 + O(ds) does not come near.
__device__ __forceinline__ float rcp(float x) { return rcp_hw(x); }
__device__ __forceinline__ double rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = __fma_rn(y, __fma_rn(-x, y, 1.0), y);
  return __fma_rn(y, __fma_rn(-x, y, 1.0), y);
}

// Local elimination of the interior rows 0..K-2 of a lane with three
// right-hand sides -- r, -a_0 at the first row, -c_{K-2} at the last row: on
// return row i is x_i + y_i u(left separator) + z_i u(own separator).
template <typename T, int K>
__device__ __forceinline__ void eliminate(const T (&a)[K], const T (&d)[K], const T (&c)[K], const T (&r)[K],
                                          T (&x)[K - 1], T (&y)[K - 1], T (&z)[K - 1], int* err) {
  T g[K - 1];
  T bet = (T)1;
#pragma unroll
  for (int i = 0; i < K - 1; ++i) {
    const int im = i > 0 ? i - 1 : 0;
    const T gi = i == 0 ? (T)0 : r_mul(c[im], bet);
    const T piv = i == 0 ? d[0] : r_fma(-a[i], gi, d[i]);
    if (piv == (T)0) atomicOr(err, 1);
    bet = rcp(piv);
    g[i] = gi;
    x[i] = r_mul(i == 0 ? r[0] : r_fma(-a[i], x[im], r[i]), bet);
    y[i] = r_mul(i == 0 ? -a[0] : r_mul(-a[i], y[im]), bet);
    const T zr = i == K - 2 ? -c[i] : (T)0;
    z[i] = r_mul(i == 0 ? zr : r_fma(-a[i], z[im], zr), bet);
  }
#pragma unroll
  for (int i = K - 3; i >= 0; --i) {
    x[i] = r_fma(-g[i + 1], x[i + 1], x[i]);
    y[i] = r_fma(-g[i + 1], y[i + 1], y[i]);
    z[i] = r_fma(-g[i + 1], z[i + 1], z[i]);
  }
}

// One line system on the G-lane group of the calling lane.  Lane l of the
// group owns K consecutive rows (rows past the line's end are identity rows
// that couple to nothing); row K-1 of each lane is its separator.  The rows
// are given as arrays of the sub-diagonal a, the diagonal d, the
// super-diagonal c and the right-hand side r; the solution u is returned in
// place of r.  `periodic`: row 0 of lane 0 couples to the last lane's
// separator through a, and that separator to row 0 through c (all G lanes
// own rows).  K is a compile-time constant so that every row stays in
// registers.  i0 = 1: the lane has K - 1 rows, entries 1 .. K - 1, and entry 0
// repeats its left neighbour (a = -1, d = 1, c = 0, r = 0); K >= 3 then.  All
// G lanes of the group must call it together.
template <int G, int K, typename T>
__device__ __forceinline__ void solve(const T (&a)[K], const T (&d)[K], const T (&c)[K],
                                      T (&r)[K], bool periodic, int* err, int i0 = 0) {
  static_assert(K >= 2, "a lane needs an interior row and a separator");
  const int lane = threadIdx.x & 31;
  const int gl = lane & (G - 1);          // lane within the group
  const int base = lane - gl;
  const unsigned mask = 0xffffffffu;
  T x[K - 1], y[K - 1], z[K - 1];
  eliminate<T, K>(a, d, c, r, x, y, z, err);
  // the separator row in its neighbours' terms: the last interior row of this
  // lane and the first interior row of the next lane
  constexpr int S = K - 1, Li = K - 2;
  const int nx = base + ((gl + 1) & (G - 1));
  constexpr int F1 = K > 2 ? 1 : 0;        // a short lane's first row
  T xn = __shfl_sync(mask, i0 ? x[F1] : x[0], nx), yn = __shfl_sync(mask, i0 ? y[F1] : y[0], nx),
    zn = __shfl_sync(mask, i0 ? z[F1] : z[0], nx);
  if (!periodic && gl == G - 1) { xn = (T)0; yn = (T)0; zn = (T)0; }
  T A = r_mul(a[S], y[Li]);
  T B = r_fma(c[S], yn, r_fma(a[S], z[Li], d[S]));
  T C = r_mul(c[S], zn);
  T R = r_fma(-c[S], xn, r_fma(-a[S], x[Li], r[S]));
  // parallel cyclic reduction over the group (identity beyond its ends
  // unless periodic)
#pragma unroll
  for (int st = 1; st < G; st *= 2) {
    const int su = base + ((gl - st) & (G - 1)), sd = base + ((gl + st) & (G - 1));
    T Au = __shfl_sync(mask, A, su), Bu = __shfl_sync(mask, B, su);
    T Cu = __shfl_sync(mask, C, su), Ru = __shfl_sync(mask, R, su);
    T Ad = __shfl_sync(mask, A, sd), Bd = __shfl_sync(mask, B, sd);
    T Cd = __shfl_sync(mask, C, sd), Rd = __shfl_sync(mask, R, sd);
    T iu = (T)0, id = (T)0;
    if constexpr (sizeof(T) == 8) {   // one reciprocal a lane, shuffled
      if (B == (T)0) atomicOr(err, 1);
      const T i0 = rcp(B);
      iu = __shfl_sync(mask, i0, su);
      id = __shfl_sync(mask, i0, sd);
    }
    if (!periodic && gl - st < 0) { Au = (T)0; Bu = (T)1; iu = (T)1; Cu = (T)0; Ru = (T)0; }
    if (!periodic && gl + st >= G) { Ad = (T)0; Bd = (T)1; id = (T)1; Cd = (T)0; Rd = (T)0; }
    if constexpr (sizeof(T) == 4) {
      if (Bu == (T)0 || Bd == (T)0) atomicOr(err, 1);
      iu = rcp(Bu);
      id = rcp(Bd);
    }
    const T kl = r_mul(A, iu);
    const T kr = r_mul(C, id);
    const T nB = r_fma(-kr, Ad, r_fma(-kl, Cu, B));
    const T nR = r_fma(-kr, Rd, r_fma(-kl, Ru, R));
    A = r_mul(-kl, Au);
    C = r_mul(-kr, Cd);
    B = nB;
    R = nR;
  }
  // after log2 G steps the reduced equation couples only to the lane itself:
  // periodic lines reach it through both neighbours, open lines never
  const T den = periodic ? r_add(r_add(A, C), B) : B;
  if (den == (T)0) atomicOr(err, 1);
  const T v = r_mul(R, rcp(den));          // u at this lane's separator
  T vl = __shfl_sync(mask, v, base + ((gl - 1) & (G - 1)));
  if (!periodic && gl == 0) vl = (T)0;
#pragma unroll
  for (int i = 0; i < K - 1; ++i) r[i] = r_fma(z[i], v, r_fma(y[i], vl, x[i]));
  r[S] = v;
}

}  // namespace fw

// ---------------------------------------------------------------------------
// 1D CN chain (Film_1D / brush, FP32 increment form, see cn_rhs) with one warp
// per (line, chain): lane l owns rows [l K, l K + K - 1] of the line's gz + 1
// rows (K = film_warp_rows; rows past the wall are identity padding), keeps
// their q in registers for the whole contour, exchanges edge values by
// shuffles, and solves each step with fw::solve.  `chain`: slices
// [(ns+1)][npts] of the chain, rows of this line at stride `stride`.
// Per-warp shared memory `sm` holds, by row: the mesh factors alpha, gamma, the
// field of types 0 and 1, and a staging row through which each finished
// slice goes to global memory (coalesced for one-line films).
// Bound: the latency of the solve's dependent operations.
// ---------------------------------------------------------------------------
constexpr int kFilmWarpM = 8;                 // rows per lane at most: lines up to 32 * 8 planes
constexpr int kFilmWarpRows = 32 * kFilmWarpM;
struct FilmWarpSm {
  float al[kFilmWarpRows], ga[kFilmWarpRows], w0[kFilmWarpRows], w1[kFilmWarpRows], stage[kFilmWarpRows];
};

// One CN row of a step: matrix and right-hand side from the mesh factors al,
// ga and the step's term w (FP32: field, FP64: beta + w / 2); qm, q0, qp: q
// of the row and its neighbours (FP64 reads q0 only).  FP64 writes the step
// (1 + ds M) q' = (1 - ds M) q as (1 + ds M) v = q, q' = 2 v - q (on the walls v
// = q / 2, so q' = 0): the right-hand side is q itself, which spares five FP64
// operations a row and the neighbours' values on GB300's narrow FP64 pipe.
template <typename T>
__device__ __forceinline__ void cn_line_row(const CnStep& st, T al, T ga, T w, T qm, T q0, T qp,
                                            T& a, T& d, T& c, T& r) {
  if constexpr (sizeof(T) == 4) {
    const float hw = __fmul_rn(st.hdsf, w);
    a = __fmul_rn(-st.dsf, al);
    c = __fmul_rn(-st.dsf, ga);
    const float b = -__fadd_rn(a, c);
    d = __fadd_rn(__fadd_rn(1.f, b), hw);
    r = cn_rhs<float>(a, b, c, hw, qm, q0, qp);
  } else {
    a = r_mul(-st.ds, al);
    c = r_mul(-st.ds, ga);
    d = r_fma(st.ds, w, 1.0);
    r = q0;
  }
}
// right-hand side of a wall row, and the new q of a row from its solution u
__device__ __forceinline__ float cn_wall_rhs(float q) { return -q; }
__device__ __forceinline__ double cn_wall_rhs(double q) { return r_mul(0.5, q); }
__device__ __forceinline__ float cn_new_q(float q, float u) { return __fadd_rn(q, u); }
__device__ __forceinline__ double cn_new_q(double q, double u) { return r_fma(2.0, u, -q); }

template <int K>
__device__ __forceinline__ void film1d_chain_warp(const FilmDev<float>& F, int dir, float* chain,
                                                  size_t stride, FilmWarpSm& sm) {
  const int lane = threadIdx.x & 31;
  const int n = F.gz + 1;
  const int s0 = lane * K;                    // this lane's rows s0 .. s0 + K - 1
  float q[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int j = s0 + i;
    float v = 0.f;
    if (j < n) v = F.single ? chain[(size_t)j * stride] : (dir == 1 && F.brush) ? (float)F.graft[j] : 1.f;
    q[i] = v;
  }
  if (!F.single) {
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (s0 + i < n) sm.stage[s0 + i] = q[i];
    __syncwarp();
    for (int j = lane; j < n; j += 32) chain[(size_t)j * stride] = sm.stage[j];
    __syncwarp();
  }
  for (int s = 1; s <= F.ns; ++s) {
    const CnStep st = cn_step(film_ds(F.dss, dir, s, F.ns));
    const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
    const float* wl = ty == 0 ? sm.w0 : sm.w1;
    // edge values of the neighbouring lanes' rows
    const float qprev = __shfl_up_sync(0xffffffffu, q[K - 1], 1);
    const float qnext = __shfl_down_sync(0xffffffffu, q[0], 1);
    float a[K], d[K], c[K], r[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = s0 + i;
      a[i] = 0.f; d[i] = 1.f; c[i] = 0.f; r[i] = 0.f;
      if (j < n) {
        if (j == 0 || j == n - 1) {
          r[i] = cn_wall_rhs(q[i]);            // Dirichlet wall: q' = 0
        } else {
          const float qm = i == 0 ? qprev : q[i > 0 ? i - 1 : 0];
          const float qp = i == K - 1 ? qnext : q[i + 1 < K ? i + 1 : i];
          cn_line_row<float>(st, sm.al[j], sm.ga[j], wl[j], qm, q[i], qp, a[i], d[i], c[i], r[i]);
        }
      }
    }
    fw::solve<32, K>(a, d, c, r, false, F.err);
    float* qn = chain + (size_t)s * F.npts;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      q[i] = cn_new_q(q[i], r[i]);
      if (s0 + i < n) sm.stage[s0 + i] = q[i];
    }
    __syncwarp();
    for (int j = lane; j < n; j += 32) qn[(size_t)j * stride] = sm.stage[j];
    __syncwarp();
  }
}

// rows per lane of an n-row line: the smallest K >= 2 with 32 K >= n
__host__ __device__ __forceinline__ int film_warp_rows(int n) { return n <= 64 ? 2 : (n + 31) / 32; }

__device__ __forceinline__ void film1d_chain_warp_any(const FilmDev<float>& F, int dir, float* chain,
                                                      size_t stride, FilmWarpSm& sm) {
  switch (film_warp_rows(F.gz + 1)) {
    case 2: film1d_chain_warp<2>(F, dir, chain, stride, sm); break;
    case 3: film1d_chain_warp<3>(F, dir, chain, stride, sm); break;
    case 4: film1d_chain_warp<4>(F, dir, chain, stride, sm); break;
    case 5: film1d_chain_warp<5>(F, dir, chain, stride, sm); break;
    case 6: film1d_chain_warp<6>(F, dir, chain, stride, sm); break;
    case 7: film1d_chain_warp<7>(F, dir, chain, stride, sm); break;
    default: film1d_chain_warp<8>(F, dir, chain, stride, sm); break;
  }
}

// mesh factors al, ga of row j and the term of field value w there (see
// cn_line_row); w32: the FP32 copy of the field value
template <typename T>
__device__ __forceinline__ T cn_mesh(const FilmDev<T>& F, int j, bool up) {
  if constexpr (sizeof(T) == 4) return up ? F.gaf[j] : F.alf[j];
  else return up ? F.gamma[j] : F.alpha[j];
}
template <typename T>
__device__ __forceinline__ T cn_term(const FilmDev<T>& F, int j, double w) {
  if constexpr (sizeof(T) == 4) return (float)w;
  else return r_fma(0.5, w, F.beta[j]);
}

// mesh factors and FP32 field of one line into the warp's shared memory;
// `field`: [ntypes][npts], rows of the line at stride `wstride`
__device__ __forceinline__ void film_warp_tables(const FilmDev<float>& F, const double* field, size_t wstride,
                                                 FilmWarpSm& sm) {
  const int lane = threadIdx.x & 31;
  for (int j = lane; j <= F.gz; j += 32) {
    sm.al[j] = F.alf[j];
    sm.ga[j] = F.gaf[j];
    sm.w0[j] = (float)field[(size_t)j * wstride];
    sm.w1[j] = F.ntypes == 2 && !F.single ? (float)field[F.npts + (size_t)j * wstride] : 0.f;
  }
  __syncwarp();
}

// Whether every system of a line's chains is diagonally dominant: 1 + ds w / 2
// >= 0.01 for the largest step and the lowest field value (the mesh terms
// are, b = |a| + |c|, unless a step goes backwards).  Then no elimination order meets a zero pivot.  Where
// it is not, the order decides which pivots vanish and how far rounding
// grows, and the chain runs the reference's serial recurrence instead
// (film_line_serial).  Every lane of a warp calls it; the answer is uniform over
// the warps of a line.
template <typename T>
__device__ __forceinline__ bool film_line_dominant(const FilmDev<T>& F, const double* field, size_t wstride) {
  if (F.backwards) return false;
  double lo = 0.0;
  const int types = F.single ? 1 : F.ntypes;
  for (int t = 0; t < types; ++t)
#pragma unroll 4
    for (int j = threadIdx.x & 31; j <= F.gz; j += 32) lo = fmin(lo, field[(size_t)t * F.npts + (size_t)j * wstride]);
#pragma unroll
  for (int o = 16; o; o >>= 1) lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
  return 1.0 + 0.5 * F.ds_max * lo >= 0.01;
}

// Whether line `line` is not for the cooperative solve.  Its chains then run the
// recurrence: here, by the thread with `lead`, where `serial` is null (a context
// of one line), else in k_film1d_chains or k_film1d_chains_sm behind this kernel,
// which take the lines that are marked in `serial` a thread each, neighbouring
// lines in neighbouring threads (2048 lines of 101 rows, a step of both chains:
// 766 us with a lane of every warp at work).
// film1d_chain as a call: inlined into the cooperative kernels it takes registers
// from their loops
template <typename T>
__device__ __noinline__ void film1d_chain_call(const FilmDev<T>& F, const double* field, int line, int dir) {
  film1d_chain<T>(F, field, line, dir);
}
template <typename T>
__device__ __forceinline__ bool film_line_serial(const FilmDev<T>& F, const double* field, int line, int dir, bool lead,
                                                 int* __restrict__ serial) {
  const bool yes = !film_line_dominant<T>(F, field + line, F.nlines);
  if (lead) {
    if (serial) {
      if (dir == 0) serial[line] = yes;
    } else if (yes) {
      film1d_chain_call<T>(F, field, line, dir);
    }
  }
  return yes;
}

// Single context (Film_1D / brush lines of one film): one warp per (line,
// chain); blockIdx.y = chain.
static __global__ void __launch_bounds__(128)
k_film1d_warp(FilmDev<float> F, FieldRef fr) {
  __shared__ FilmWarpSm sm_all[4];
  const int wib = threadIdx.x >> 5;
  const int line = blockIdx.x * 4 + wib;
  if (line >= F.nlines) return;
  const int dir = blockIdx.y;
  const size_t L = F.nlines;
  FilmWarpSm& sm = sm_all[wib];
  film_warp_tables(F, fr.get() + line, L, sm);
  film1d_chain_warp_any(F, dir, (dir == 0 ? F.q : F.qd) + line, L, sm);
}

// Batch: one warp per (film, chain) of `items` ((film << 1) | chain, longest
// contours first), the field from the film's current SCF history slot.
static __global__ void __launch_bounds__(128)
k_film1d_warp_b(const FilmDev<float>* __restrict__ Fs, const ScfDev* __restrict__ Ss,
                const int* __restrict__ items, int nitems) {
  __shared__ FilmWarpSm sm_all[4];
  const int wib = threadIdx.x >> 5;
  const int it = blockIdx.x * 4 + wib;
  if (it >= nitems) return;
  const int f = items[it] >> 1, dir = items[it] & 1;
  const FilmDev<float> F = Fs[f];
  const ScfDev& S = Ss[f];
  const double* field = S.hx + (size_t)((*S.iter) % S.slots) * ((size_t)S.ntypes * S.npts);
  FilmWarpSm& sm = sm_all[wib];
  film_warp_tables(F, field, 1, sm);
  film1d_chain_warp_any(F, dir, dir == 0 ? F.q : F.qd, 1, sm);
}

// ---------------------------------------------------------------------------
// Longer lines (FP32 257 .. 4096 rows, FP64 1025 .. 4096, film_line.cuh has the
// shorter ones): W warps per (line, chain), K = 4 rows per lane, W the power of two >= rows / 128.  Each warp reduces its 128 rows to
// one equation in the last rows of itself and its neighbours:
//  - lanes eliminate their interior rows (fw::eliminate), then the warp's 31
//    first separators by cyclic reduction with the warp's two boundary
//    unknowns as extra right-hand sides, so every row of the warp is
//    x + y U(previous warp) + z U(this warp), U = solution at a warp's last row;
//  - the warps exchange seven numbers each (their last row's equation and
//    their first row's x, y, z; ten in FP32, see FilmGroupSm) and every warp solves the W equations in U
//    itself, one lane per equation: one barrier per contour step.
// The exchange slots are double buffered by step parity: a warp writes the
// slots of step s + 2 only after the barrier of step s + 1, which every warp
// passes after its reads of step s.
//
// A single line puts its warps in different CTAs of a cluster (at most 8),
// since FP64 instructions of warps on one SM share one narrow pipe: the
// exchange goes to every CTA's shared memory and the barrier is the
// cluster's.  Many lines keep their warps in one CTA (clusters of one).  The
// arithmetic is the same either way: K and W depend on the line length alone.
// Bound: FP64 issue, one warp instruction per 64 cycles on each SM quarter.
// Measured (GB300, one line, against one thread per line and chain; a step of
// both chains): FP64 2001 rows 2290 -> 17 us; FP32 301 rows 52 -> 8.6 us, 1001
// rows 157 -> 9.6.
// ---------------------------------------------------------------------------
constexpr int kFilmGroupK = 4;
constexpr int kFilmGroupMaxW = 32;
constexpr int kFilmGroupRows = kFilmGroupMaxW * 32 * kFilmGroupK;
__host__ __device__ __forceinline__ int film_group_warps(int n) {
  int w = 2;
  while (w * 32 * kFilmGroupK < n) w *= 2;
  return w;
}

namespace fw {

__device__ __forceinline__ unsigned cluster_map(const void* p, int rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_store(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace fw

// What the warps exchange a step, by step parity: A, B, R, c of their last
// row's equation and x0, y0, z0 of their first row.  FP32 forms the next
// step's right-hand side from differences of q, with its own copy of the next
// warp's first q: it takes the six numbers that row is made of there (x, y, z of
// the row, X, Y, Z of its separator), so that the copy never differs from the
// row.  A copy that rounds on its own drifts, and ds / dz^2 times the drift is
// a source at every warp's edge (1501 rows, 1200 steps: density 1e-5 off).
template <typename T>
struct FilmGroupSm {
  static constexpr int kN = sizeof(T) == 4 ? 10 : 7;
  T ex[2][kN][kFilmGroupMaxW];
};

// `chain`, `stride`, `field`, `wstride` as film1d_chain_warp / film_warp_tables;
// csize: CTAs of the cluster, W = csize * (blockDim.x / 32) warps.
template <typename T>
__device__ __forceinline__ void film1d_chain_group(const FilmDev<T>& F, int dir, T* chain, size_t stride,
                                                   const double* field, size_t wstride, int crank, int csize,
                                                   FilmGroupSm<T>& sm) {
  constexpr int K = kFilmGroupK, S = K - 1, Li = K - 2;
  const unsigned mask = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int W = csize * (blockDim.x >> 5);
  const int w = crank * (blockDim.x >> 5) + (threadIdx.x >> 5);   // this warp of the line
  const int n = F.gz + 1;
  const int s0 = (w * 32 + lane) * K;
  T q[K], al[K], ga[K], t0[K], t1[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int j = s0 + i;
    T v = (T)0;
    al[i] = ga[i] = t0[i] = t1[i] = (T)0;
    if (j < n) {
      v = F.single ? chain[(size_t)j * stride] : (dir == 1 && F.brush) ? (T)F.graft[j] : (T)1;
      al[i] = cn_mesh<T>(F, j, false);
      ga[i] = cn_mesh<T>(F, j, true);
      t0[i] = cn_term<T>(F, j, field[(size_t)j * wstride]);
      if (F.ntypes == 2 && !F.single) t1[i] = cn_term<T>(F, j, field[F.npts + (size_t)j * wstride]);
      if (!F.single) chain[(size_t)j * stride] = v;
    }
    q[i] = v;
  }
  // FP32: q of the previous warp's last row and the next warp's first row
  T qlo = (T)0, qhi = (T)0;
  if constexpr (sizeof(T) == 4) {
    auto q0_of = [&](int j) {
      if (j < 0 || j >= n) return (T)0;
      return F.single ? chain[(size_t)j * stride] : (dir == 1 && F.brush) ? (T)F.graft[j] : (T)1;
    };
    qlo = q0_of(w * 32 * K - 1);
    qhi = q0_of((w + 1) * 32 * K);
  }
  for (int s = 1; s <= F.ns; ++s) {
    const CnStep st = cn_step(film_ds(F.dss, dir, s, F.ns));
    const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
    T qprev = (T)0, qnext = (T)0;
    if constexpr (sizeof(T) == 4) {
      qprev = __shfl_up_sync(mask, q[K - 1], 1);
      qnext = __shfl_down_sync(mask, q[0], 1);
      if (lane == 0) qprev = qlo;
      if (lane == 31) qnext = qhi;
    }
    T a[K], d[K], c[K], r[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = s0 + i;
      a[i] = (T)0; d[i] = (T)1; c[i] = (T)0; r[i] = (T)0;
      if (j < n) {
        if (j == 0 || j == n - 1) {
          r[i] = cn_wall_rhs(q[i]);
        } else {
          const T qm = i == 0 ? qprev : q[i > 0 ? i - 1 : 0];
          const T qp = i == K - 1 ? qnext : q[i + 1 < K ? i + 1 : i];
          cn_line_row<T>(st, al[i], ga[i], ty == 0 ? t0[i] : t1[i], qm, q[i], qp, a[i], d[i], c[i], r[i]);
        }
      }
    }
    T x[K - 1], y[K - 1], z[K - 1];
    fw::eliminate<T, K>(a, d, c, r, x, y, z, F.err);
    // separator equations of lanes 0..30 in the warp's boundary unknowns:
    // lane 0's left neighbour is the previous warp's last row (right-hand
    // side Y), lane 30's right neighbour this warp's last row (Z); lane 31
    // takes no part (identity)
    const T xn = __shfl_down_sync(mask, x[0], 1), yn = __shfl_down_sync(mask, y[0], 1),
            zn = __shfl_down_sync(mask, z[0], 1);
    const T As = r_mul(a[S], y[Li]);
    const T Bs = r_fma(a[S], z[Li], d[S]);
    const T Rs = r_fma(-a[S], x[Li], r[S]);
    T A = As, B = r_fma(c[S], yn, Bs), C = r_mul(c[S], zn), R = r_fma(-c[S], xn, Rs), Y = (T)0, Z = (T)0;
    if (lane == 0) { Y = -A; A = (T)0; }
    if (lane == 30) { Z = -C; C = (T)0; }
    if (lane == 31) { A = (T)0; B = (T)1; C = (T)0; R = (T)0; }
#pragma unroll
    for (int sp = 1; sp < 32; sp *= 2) {
      if (B == (T)0) atomicOr(F.err, 1);
      const T iB = fw::rcp(B);
      const int su = (lane - sp) & 31, sd = (lane + sp) & 31;
      T Au = __shfl_sync(mask, A, su), Iu = __shfl_sync(mask, iB, su), Cu = __shfl_sync(mask, C, su);
      T Ru = __shfl_sync(mask, R, su), Yu = __shfl_sync(mask, Y, su), Zu = __shfl_sync(mask, Z, su);
      T Ad = __shfl_sync(mask, A, sd), Id = __shfl_sync(mask, iB, sd), Cd = __shfl_sync(mask, C, sd);
      T Rd = __shfl_sync(mask, R, sd), Yd = __shfl_sync(mask, Y, sd), Zd = __shfl_sync(mask, Z, sd);
      // beyond the ends A or C is zero, so the wrapped values drop out
      const T kl = r_mul(A, Iu), kr = r_mul(C, Id);
      B = r_fma(-kr, Ad, r_fma(-kl, Cu, B));
      R = r_fma(-kr, Rd, r_fma(-kl, Ru, R));
      Y = r_fma(-kr, Yd, r_fma(-kl, Yu, Y));
      Z = r_fma(-kr, Zd, r_fma(-kl, Zu, Z));
      A = r_mul(-kl, Au);
      C = r_mul(-kr, Cd);
    }
    if (B == (T)0) atomicOr(F.err, 1);
    const T iB = fw::rcp(B);
    T X = r_mul(R, iB);
    Y = r_mul(Y, iB);
    Z = r_mul(Z, iB);
    if (lane == 31) { X = (T)0; Y = (T)0; Z = (T)1; }   // its separator is U itself
    // the warp's numbers: its last row's equation (lane 31, in the terms of
    // lane 30's separator) and its first row (lane 0)
    const T X30 = __shfl_sync(mask, X, 30), Y30 = __shfl_sync(mask, Y, 30), Z30 = __shfl_sync(mask, Z, 30);
    const T eA = __shfl_sync(mask, r_mul(As, Y30), 31), eB = __shfl_sync(mask, r_fma(As, Z30, Bs), 31);
    const T eR = __shfl_sync(mask, r_fma(-As, X30, Rs), 31), eC = __shfl_sync(mask, c[S], 31);
    T (*ex)[kFilmGroupMaxW] = sm.ex[s & 1];
    if constexpr (sizeof(T) == 4) {       // one CTA
      if (lane == 0) {
        ex[0][w] = eA; ex[1][w] = eB; ex[2][w] = eR; ex[3][w] = eC;
        ex[4][w] = x[0]; ex[5][w] = y[0]; ex[6][w] = z[0];
        ex[7][w] = X; ex[8][w] = Y; ex[9][w] = Z;
      }
    } else {
      const T fx = __shfl_sync(mask, r_fma(z[0], X, x[0]), 0), fy = __shfl_sync(mask, r_fma(z[0], Y, y[0]), 0);
      const T fz = __shfl_sync(mask, r_mul(z[0], Z), 0);
      for (int k = lane; k < 7 * csize; k += 32) {
        const int which = k % 7, to = k / 7;
        const T v = which == 0 ? eA : which == 1 ? eB : which == 2 ? eR : which == 3 ? eC : which == 4 ? fx : which == 5 ? fy : fz;
        if (csize == 1) ex[which][w] = v;
        else fw::cluster_store(fw::cluster_map(&ex[which][w], to), v);
      }
    }
    if (csize == 1) __syncthreads();
    else fw::cluster_barrier();
    // every warp solves the W equations, lane l the one of warp l
    T gA = (T)0, gB = (T)1, gC = (T)0, gR = (T)0, hx = (T)0, hy = (T)0, hz = (T)0;
    if (lane < W) {
      gA = ex[0][lane]; gB = ex[1][lane]; gR = ex[2][lane];
      if (lane + 1 < W) {
        hx = ex[4][lane + 1]; hy = ex[5][lane + 1]; hz = ex[6][lane + 1];
        if constexpr (sizeof(T) == 4) {
          hx = r_fma(hz, ex[7][lane + 1], hx);
          hy = r_fma(hz, ex[8][lane + 1], hy);
          hz = r_mul(hz, ex[9][lane + 1]);
        }
      }
      const T cc = ex[3][lane];
      gB = r_fma(cc, hy, gB);
      gR = r_fma(-cc, hx, gR);
      gC = r_mul(cc, hz);
      if (lane == 0) gA = (T)0;
    }
    for (int sp = 1; sp < W; sp *= 2) {
      if (gB == (T)0) atomicOr(F.err, 1);
      const T i0 = fw::rcp(gB);
      const int su = (lane - sp) & 31, sd = (lane + sp) & 31;
      const T Au = __shfl_sync(mask, gA, su), Iu = __shfl_sync(mask, i0, su), Cu = __shfl_sync(mask, gC, su),
              Ru = __shfl_sync(mask, gR, su);
      const T Ad = __shfl_sync(mask, gA, sd), Id = __shfl_sync(mask, i0, sd), Cd = __shfl_sync(mask, gC, sd),
              Rd = __shfl_sync(mask, gR, sd);
      const T kl = r_mul(gA, Iu), kr = r_mul(gC, Id);
      gB = r_fma(-kr, Ad, r_fma(-kl, Cu, gB));
      gR = r_fma(-kr, Rd, r_fma(-kl, Ru, gR));
      gA = r_mul(-kl, Au);
      gC = r_mul(-kr, Cd);
    }
    if (gB == (T)0) atomicOr(F.err, 1);
    const T U = r_mul(gR, fw::rcp(gB));
    const T UL = w > 0 ? __shfl_sync(mask, U, w > 0 ? w - 1 : 0) : (T)0;
    const T UR = __shfl_sync(mask, U, w);
    // separators of the lanes, then their interior rows
    const T v = r_fma(Z, UR, r_fma(Y, UL, X));
    T vl = __shfl_up_sync(mask, v, 1);
    if (lane == 0) vl = UL;
    T* qn = chain + (size_t)s * F.npts;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const T u = i == S ? v : r_fma(z[i < S ? i : 0], v, r_fma(y[i < S ? i : 0], vl, x[i < S ? i : 0]));
      q[i] = cn_new_q(q[i], u);
      if (s0 + i < n) qn[(size_t)(s0 + i) * stride] = q[i];
    }
    if constexpr (sizeof(T) == 4) {   // the neighbouring warps' edge rows, by those warps' own operations
      qlo = cn_new_q(qlo, UL);
      if (w + 1 < W) {
        const T UN = __shfl_sync(mask, U, w + 1);
        const T vn = r_fma(ex[9][w + 1], UN, r_fma(ex[8][w + 1], UR, ex[7][w + 1]));
        qhi = cn_new_q(qhi, r_fma(ex[6][w + 1], vn, r_fma(ex[5][w + 1], UR, ex[4][w + 1])));
      }
    }
  }
}

// Single context: clusters of csize CTAs, one cluster per line; blockIdx.y =
// chain.  MAXT: 256 threads keep every value of an FP64 row in registers,
// 1024 (lines of more than 1024 rows in one CTA) spill some.
template <typename T, int MAXT>
__global__ void __launch_bounds__(MAXT)
k_film1d_group(FilmDev<T> F, FieldRef fr, int csize, int* __restrict__ serial) {
  __shared__ FilmGroupSm<T> sm;
  if (csize > 1) fw::cluster_barrier();   // every CTA of the cluster runs before its memory is written
  const int line = blockIdx.x / csize, dir = blockIdx.y;
  const size_t L = F.nlines;
  if (film_line_serial<T>(F, fr.get(), line, dir, threadIdx.x == 0 && blockIdx.x % csize == 0, serial)) return;
  film1d_chain_group<T>(F, dir, (dir == 0 ? F.q : F.qd) + line, L, fr.get() + line, L, blockIdx.x % csize, csize, sm);
}

// Batch: one CTA per (film, chain) of `items`, all with blockDim.x / 32 warps
// per line.
template <typename T, int MAXT>
__global__ void __launch_bounds__(MAXT)
k_film1d_group_b(const FilmDev<T>* __restrict__ Fs, const ScfDev* __restrict__ Ss, const int* __restrict__ items,
                 int* __restrict__ serial) {
  __shared__ FilmGroupSm<T> sm;
  const int f = items[blockIdx.x] >> 1, dir = items[blockIdx.x] & 1;
  const FilmDev<T> F = Fs[f];
  const ScfDev& S = Ss[f];
  const double* field = S.hx + (size_t)((*S.iter) % S.slots) * ((size_t)S.ntypes * S.npts);
  if (film_line_serial<T>(F, field, 0, dir, threadIdx.x == 0, serial + f)) return;
  film1d_chain_group<T>(F, dir, dir == 0 ? F.q : F.qd, 1, field, 1, 0, 1, sm);
}

// ---------------------------------------------------------------------------
// Douglas ADI sweeps (Film_CK_AD/Film_3D/Geometry_Modules/mod_realspace.f90:
// 22-140) in FP32 increment form with the warp solver: G lanes per line, K
// consecutive points per lane (G K = gx or gy for the periodic x and y lines;
// G K >= gz + 1 for the Dirichlet z lines, padded with identity rows), 32 / G
// lines per warp.  Same right-hand sides as k_adi_x / k_adi_y / k_adi_z; the
// x and y systems are the reference's periodic ones (cyclicTriDiag, :149-176)
// solved with the reduced system closed cyclically.  blockIdx.y = chain.
// ---------------------------------------------------------------------------
// Shape of a warp-solver sweep: G lanes per line, K points per lane (g = 0:
// the one-thread-per-line kernels); staged: the tile goes through shared
// memory (k_adi_yz_s, y and z sweeps).
struct AdiShape {
  int g, k, staged;
};

// Per-chain FP32 coefficients of a step, read from the context's table
// (formed in FP64 on the host, rounded as k_adi_x / k_adi_y form them per
// thread): forming them on the device would keep GB300's narrow FP64 pipe
// and a block barrier on every sweep's critical path.
struct AdiCoef {
  float ax, bx, ay, by, dsf, hdsf;
};
__device__ __forceinline__ AdiCoef adi_coef(const FilmDev<float>& F, int dir, int s) {
  const float* c = F.adicf + 6 * (dir == 0 ? s : F.ns + 1 - s);
  return AdiCoef{__ldg(c), __ldg(c + 1), __ldg(c + 2), __ldg(c + 3), __ldg(c + 4), __ldg(c + 5)};
}

template <int G, int K>
__global__ void __launch_bounds__(128)
k_adi_x_w(FilmDev<float> F, int s) {
  constexpr int LPW = 32 / G;
  const int gx = F.gx, gy = F.gy, gz = F.gz, L = F.nlines;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const int id = (blockIdx.x * 4 + (threadIdx.x >> 5)) * LPW + lane / G;   // line (y, z interior)
  const int dir = blockIdx.y;
  const bool live = id < gy * (gz - 1);
  const int y = live ? id % gy : 0, z = live ? 1 + id / gy : 1;
  const AdiCoef cf = adi_coef(F, dir, s);
  const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
  const float* p0 = (dir == 0 ? F.q : F.qd) + (size_t)(s - 1) * F.npts;
  float* out = F.w1 + (size_t)dir * F.npts;
  const float* wf = F.wf + (size_t)ty * F.npts;
  const float ax = cf.ax, bx = cf.bx, cx = ax;
  const float ay = cf.ay, cy = ay;
  // z couplings as the z sweep forms them (cn_row, FP32 mesh factors)
  const float az = __fmul_rn(-cf.dsf, F.alf[z]), cz = __fmul_rn(-cf.dsf, F.gaf[z]);
  const int ym = (y + gy - 1) % gy, yp = (y + 1) % gy;
  const size_t row = (size_t)z * L + (size_t)y * gx, rym = (size_t)z * L + (size_t)ym * gx,
               ryp = (size_t)z * L + (size_t)yp * gx, rzm = row - L, rzp = row + L;
  const int x0 = gl * K;
  float c0[K];
#pragma unroll
  for (int i = 0; i < K; ++i) c0[i] = live ? __ldg(p0 + row + x0 + i) : 0.f;
  const int base = lane - gl;
  const float left = __shfl_sync(0xffffffffu, c0[K - 1], base + ((gl - 1) & (G - 1)));
  const float right = __shfl_sync(0xffffffffu, c0[0], base + ((gl + 1) & (G - 1)));
  float a[K], d[K], c[K], r[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int x = x0 + i;
    const float qxm = i == 0 ? left : c0[i > 0 ? i - 1 : 0];
    const float qxp = i == K - 1 ? right : c0[i + 1 < K ? i + 1 : i];
    float qym = 0.f, qyp = 0.f, qzm = 0.f, qzp = 0.f, dsw = 0.f;
    if (live) {
      qym = __ldg(p0 + rym + x); qyp = __ldg(p0 + ryp + x);
      qzm = __ldg(p0 + rzm + x); qzp = __ldg(p0 + rzp + x);
      dsw = cf.dsf * wf[row + x];
    }
    const float q0 = c0[i];
    r[i] = -2.f * (ax * (qxm - q0) + cx * (qxp - q0) + ay * (qym - q0) + cy * (qyp - q0) +
                   az * (qzm - q0) + cz * (qzp - q0)) - dsw * q0;
    a[i] = ax; c[i] = cx; d[i] = 1.f + bx;
  }
  fw::solve<G, K>(a, d, c, r, true, F.err);
  if (live) {
#pragma unroll
    for (int i = 0; i < K; ++i) out[row + x0 + i] = c0[i] + r[i];
  }
}

template <int G, int K>
__global__ void __launch_bounds__(128)
k_adi_y_w(FilmDev<float> F, int s) {
  constexpr int LPW = 32 / G;
  const int gx = F.gx, gy = F.gy, gz = F.gz, L = F.nlines;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const int id = (blockIdx.x * 4 + (threadIdx.x >> 5)) * LPW + lane / G;   // line (x, z interior)
  const int dir = blockIdx.y;
  const bool live = id < gx * (gz - 1);
  const int x = live ? id % gx : 0, z = live ? 1 + id / gx : 1;
  const AdiCoef cf = adi_coef(F, dir, s);
  const float* p0 = (dir == 0 ? F.q : F.qd) + (size_t)(s - 1) * F.npts;
  float* w1 = F.w1 + (size_t)dir * F.npts;
  const float ay = cf.ay, by = cf.by, cy = ay;
  const size_t col = (size_t)z * L + x;
  const int y0 = gl * K;
  // e = q - q* at the lane's points; q* kept for the write-back
  float e[K], ws[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const size_t idx = col + (size_t)(y0 + i) * gx;
    ws[i] = live ? w1[idx] : 0.f;
    e[i] = live ? __ldg(p0 + idx) - ws[i] : 0.f;
  }
  const int base = lane - gl;
  const float left = __shfl_sync(0xffffffffu, e[K - 1], base + ((gl - 1) & (G - 1)));
  const float right = __shfl_sync(0xffffffffu, e[0], base + ((gl + 1) & (G - 1)));
  float a[K], d[K], c[K], r[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const float em = i == 0 ? left : e[i > 0 ? i - 1 : 0];
    const float ep = i == K - 1 ? right : e[i + 1 < K ? i + 1 : i];
    r[i] = ay * (em - e[i]) + cy * (ep - e[i]);
    a[i] = ay; c[i] = cy; d[i] = 1.f + by;
  }
  fw::solve<G, K>(a, d, c, r, true, F.err);
  if (live) {
#pragma unroll
    for (int i = 0; i < K; ++i) w1[col + (size_t)(y0 + i) * gx] = ws[i] + r[i];
  }
}

// x and y sweeps of one interior plane in one block (gx = gy = N = G K, all N
// lines of a sweep at once: N G threads).  The plane of the previous slice
// and the x sweep's result stay in shared memory ([y][x]), so the y sweep
// reads no global memory and the plane leaves once, row by row.  Right-hand
// sides, matrices and solver are those of k_adi_x_w and k_adi_y_w with the
// same shape, operation for operation; the neighbouring planes z - 1 and
// z + 1 (the x sweep's z couplings) are read from global memory as there.
// grid (gz - 1 planes, chains).
template <int G, int K>
__global__ void __launch_bounds__(G * K * G, 1)
k_adi_xy_p(FilmDev<float> F, int s) {
  constexpr int N = G * K;                 // points of an x or a y line
  constexpr int LPW = 32 / G;              // lines per warp
  static_assert(N * G <= 1024 && N % LPW == 0, "one block holds every line of the plane");
  __shared__ float P[N * N];               // previous slice, plane z
  __shared__ float Wp[N * N];              // x sweep's result, then the y sweep's
  const int L = F.nlines;                  // = N * N
  const int z = 1 + blockIdx.x, dir = blockIdx.y;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const int line = (threadIdx.x >> 5) * LPW + lane / G;   // y for the x sweep, x for the y sweep
  const AdiCoef cf = adi_coef(F, dir, s);
  const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
  const float* p0 = (dir == 0 ? F.q : F.qd) + (size_t)(s - 1) * F.npts;
  float* out = F.w1 + (size_t)dir * F.npts;
  const float* wf = F.wf + (size_t)ty * F.npts;
  const size_t pz = (size_t)z * L;
  for (int i = threadIdx.x; i < N * N; i += blockDim.x) P[i] = __ldg(p0 + pz + i);
  __syncthreads();
  const int base = lane - gl;
  {  // x sweep: line y, lane points x0 .. x0 + K - 1
    const int y = line, x0 = gl * K;
    const float ax = cf.ax, bx = cf.bx, cx = ax;
    const float ay = cf.ay, cy = ay;
    const float az = __fmul_rn(-cf.dsf, F.alf[z]), cz = __fmul_rn(-cf.dsf, F.gaf[z]);
    const int ym = (y + N - 1) % N, yp = (y + 1) % N;
    const size_t row = pz + (size_t)y * N, rzm = row - L, rzp = row + L;
    float c0[K];
#pragma unroll
    for (int i = 0; i < K; ++i) c0[i] = P[y * N + x0 + i];
    const float left = __shfl_sync(0xffffffffu, c0[K - 1], base + ((gl - 1) & (G - 1)));
    const float right = __shfl_sync(0xffffffffu, c0[0], base + ((gl + 1) & (G - 1)));
    float a[K], d[K], c[K], r[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int x = x0 + i;
      const float qxm = i == 0 ? left : c0[i > 0 ? i - 1 : 0];
      const float qxp = i == K - 1 ? right : c0[i + 1 < K ? i + 1 : i];
      const float qym = P[ym * N + x], qyp = P[yp * N + x];
      const float qzm = __ldg(p0 + rzm + x), qzp = __ldg(p0 + rzp + x);
      const float dsw = cf.dsf * wf[row + x];
      const float q0 = c0[i];
      r[i] = -2.f * (ax * (qxm - q0) + cx * (qxp - q0) + ay * (qym - q0) + cy * (qyp - q0) +
                     az * (qzm - q0) + cz * (qzp - q0)) - dsw * q0;
      a[i] = ax; c[i] = cx; d[i] = 1.f + bx;
    }
    fw::solve<G, K>(a, d, c, r, true, F.err);
#pragma unroll
    for (int i = 0; i < K; ++i) Wp[y * N + x0 + i] = c0[i] + r[i];
  }
  __syncthreads();
  {  // y sweep: line x, lane points y0 .. y0 + K - 1; each lane rewrites only its own points
    const int x = line, y0 = gl * K;
    const float ay = cf.ay, by = cf.by, cy = ay;
    float e[K], ws[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      ws[i] = Wp[(y0 + i) * N + x];
      e[i] = P[(y0 + i) * N + x] - ws[i];
    }
    const float left = __shfl_sync(0xffffffffu, e[K - 1], base + ((gl - 1) & (G - 1)));
    const float right = __shfl_sync(0xffffffffu, e[0], base + ((gl + 1) & (G - 1)));
    float a[K], d[K], c[K], r[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const float em = i == 0 ? left : e[i > 0 ? i - 1 : 0];
      const float ep = i == K - 1 ? right : e[i + 1 < K ? i + 1 : i];
      r[i] = ay * (em - e[i]) + cy * (ep - e[i]);
      a[i] = ay; c[i] = cy; d[i] = 1.f + by;
    }
    fw::solve<G, K>(a, d, c, r, true, F.err);
#pragma unroll
    for (int i = 0; i < K; ++i) Wp[(y0 + i) * N + x] = ws[i] + r[i];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N * N; i += blockDim.x) out[pz + i] = Wp[i];
}

template <int G, int K>
__global__ void __launch_bounds__(128)
k_adi_z_w(FilmDev<float> F, int s) {
  constexpr int LPW = 32 / G;
  const int gz = F.gz, L = F.nlines, n = gz + 1;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const int line0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * LPW + lane / G;
  const int dir = blockIdx.y;
  const bool live = line0 < L;
  const int line = live ? line0 : 0;
  const AdiCoef cf = adi_coef(F, dir, s);
  const CnStep st{0.0, cf.dsf, cf.hdsf};
  const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
  const float* wl = F.wf + (size_t)ty * F.npts;
  const float* p0 = (dir == 0 ? F.q : F.qd) + (size_t)(s - 1) * F.npts;
  const float* w1 = F.w1 + (size_t)dir * F.npts;
  float* qn = (dir == 0 ? F.q : F.qd) + (size_t)s * F.npts;
  const int j0 = gl * K;
  // f = q - q** (q** = 0 on the walls); q** kept for the write-back
  float f[K], wq[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int j = j0 + i;
    const size_t idx = (size_t)j * L + line;
    const bool in = live && j < n;
    const bool wall = j == 0 || j == n - 1;
    wq[i] = in && !wall ? __ldg(w1 + idx) : 0.f;
    f[i] = in ? __ldg(p0 + idx) - wq[i] : 0.f;
  }
  const int base = lane - gl;
  const float fprev = __shfl_sync(0xffffffffu, f[K - 1], base + ((gl - 1) & (G - 1)));
  const float fnext = __shfl_sync(0xffffffffu, f[0], base + ((gl + 1) & (G - 1)));
  float a[K], d[K], c[K], r[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int j = j0 + i;
    a[i] = 0.f; d[i] = 1.f; c[i] = 0.f; r[i] = 0.f;
    if (j > 0 && j < n - 1) {
      const float fm = i == 0 ? fprev : f[i > 0 ? i - 1 : 0];
      const float fp = i == K - 1 ? fnext : f[i + 1 < K ? i + 1 : i];
      float ai, ci, bi, hw;
      cn_row<float>(F, st, j, 0.0, live ? wl[(size_t)j * L + line] : 0.f, ai, ci, bi, hw);
      a[i] = ai; c[i] = ci;
      d[i] = 1.f + bi + hw;
      r[i] = ai * (fm - f[i]) + ci * (fp - f[i]) + hw * f[i];
    }
  }
  fw::solve<G, K>(a, d, c, r, false, F.err);
  if (live) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = j0 + i;
      if (j < n) qn[(size_t)j * L + line] = (j > 0 && j < n - 1) ? wq[i] + r[i] : r[i];
    }
  }
}

// ---------------------------------------------------------------------------
// Shared-memory staged y and z sweeps.  The y lines (stride gx) and z lines
// (stride gx gy) run across x, so a warp that holds one line reads a
// different 32-byte sector per lane.  Here a block takes a tile of 32
// neighbouring lines (32 consecutive x of one plane for y, 32 consecutive
// (y, x) lines for z), reads every row of the tile with 32 consecutive
// floats per warp load, keeps the tile in shared memory (rows padded to 33
// floats), solves its lines there with the warp solver (G lanes, K rows per
// lane, 128 / G lines per round of the block's four warps) and writes the
// tile back the same way.  Right-hand sides, matrices and the solver are
// those of k_adi_y_w / k_adi_z_w; neighbour values come from shared memory
// instead of shuffles.  Shared memory: (Z ? 3 : 2) n 33 floats.
// ---------------------------------------------------------------------------
constexpr int kAdiTile = 32;
constexpr int kAdiPad = 33;

__host__ __device__ constexpr size_t adi_staged_smem(int n, bool z) {
  return (size_t)(z ? 3 : 2) * n * kAdiPad * sizeof(float);
}

template <int G, int K, bool Z>
__global__ void __launch_bounds__(128)
k_adi_yz_s(FilmDev<float> F, int s) {
  static_assert(G >= 4, "four warps cover 32 lines per round at G >= 4");
  extern __shared__ __align__(16) float smf[];
  constexpr int LPW = 32 / G;
  const int gx = F.gx, L = F.nlines;
  const int n = Z ? F.gz + 1 : F.gy;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, gl = lane & (G - 1);
  size_t base, rstride;
  int cnt;
  if (Z) {
    const int l0 = blockIdx.x * kAdiTile;
    base = (size_t)l0;
    rstride = (size_t)L;
    cnt = min(kAdiTile, L - l0);
  } else {
    const int tx = (gx + kAdiTile - 1) / kAdiTile;
    const int z = 1 + blockIdx.x / tx, x0 = (blockIdx.x % tx) * kAdiTile;
    base = (size_t)z * L + x0;
    rstride = (size_t)gx;
    cnt = min(kAdiTile, gx - x0);
  }
  const int dir = blockIdx.y;
  const AdiCoef cf = adi_coef(F, dir, s);
  const float* p0 = (dir == 0 ? F.q : F.qd) + (size_t)(s - 1) * F.npts;
  float* w1 = F.w1 + (size_t)dir * F.npts;
  const int ty = (F.brush || F.single) ? 0 : film_type(dir, s, F.ns, F.na);
  const float* wl = F.wf + (size_t)ty * F.npts;
  float* sf = smf;                       // q - q** (z) or q - q* (y); then the result
  float* sw = smf + n * kAdiPad;         // q** (z, 0 on the walls) or q*
  float* sl = smf + 2 * n * kAdiPad;     // z: field of the step's type
  for (int j = wp; j < n; j += 4) {
    float f = 0.f, wq = 0.f, wv = 0.f;
    if (lane < cnt) {
      const size_t idx = base + (size_t)j * rstride + lane;
      if (Z) {
        wq = (j == 0 || j == n - 1) ? 0.f : __ldg(w1 + idx);
        wv = __ldg(wl + idx);
      } else {
        wq = w1[idx];
      }
      f = __ldg(p0 + idx) - wq;
    }
    sf[j * kAdiPad + lane] = f;
    sw[j * kAdiPad + lane] = wq;
    if (Z) sl[j * kAdiPad + lane] = wv;
  }
  __syncthreads();
  const CnStep st{0.0, cf.dsf, cf.hdsf};
  const float ay = cf.ay, by = cf.by, cy = ay;
#pragma unroll 1
  for (int r0 = 0; r0 < kAdiTile; r0 += 4 * LPW) {
    const int tl = r0 + wp * LPW + lane / G;   // line of the tile
    const int j0 = gl * K;
    float a[K], d[K], c[K], r[K], wq[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = j0 + i;
      a[i] = 0.f; d[i] = 1.f; c[i] = 0.f; r[i] = 0.f; wq[i] = 0.f;
      if (j < n) {
        const float f = sf[j * kAdiPad + tl];
        wq[i] = sw[j * kAdiPad + tl];
        if (Z) {
          if (j > 0 && j < n - 1) {
            const float fm = sf[(j - 1) * kAdiPad + tl], fp = sf[(j + 1) * kAdiPad + tl];
            float ai, ci, bi, hw;
            cn_row<float>(F, st, j, 0.0, sl[j * kAdiPad + tl], ai, ci, bi, hw);
            a[i] = ai; c[i] = ci;
            d[i] = 1.f + bi + hw;
            r[i] = ai * (fm - f) + ci * (fp - f) + hw * f;
          }
        } else {
          const float em = sf[(j == 0 ? n - 1 : j - 1) * kAdiPad + tl];
          const float ep = sf[(j == n - 1 ? 0 : j + 1) * kAdiPad + tl];
          r[i] = ay * (em - f) + cy * (ep - f);
          a[i] = ay; c[i] = cy; d[i] = 1.f + by;
        }
      }
    }
    fw::solve<G, K>(a, d, c, r, !Z, F.err);
    __syncwarp();   // every lane of the line has read its rows
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = j0 + i;
      if (j < n) sf[j * kAdiPad + tl] = (!Z || (j > 0 && j < n - 1)) ? wq[i] + r[i] : r[i];
    }
  }
  __syncthreads();
  float* out = Z ? (dir == 0 ? F.q : F.qd) + (size_t)s * F.npts : w1;
  if (lane < cnt)
    for (int j = wp; j < n; j += 4) out[base + (size_t)j * rstride + lane] = sf[j * kAdiPad + lane];
}

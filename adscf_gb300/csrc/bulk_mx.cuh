// bulk_mx.cuh -- mixed-radix line passes of the bulk propagator for grids the
// register FFT does not cover (lines of 2, 3 and 5 factors, unequal axes,
// two-dimensional grids), and for FP64 grids too small to fill the GPU there.
//
// Same double step as bulk_kernels.cuh (X, Yf, Z, Yi).  A line of
// n = R_1 R_2 ... R_S points is transformed in place in shared memory, one
// stage per radix: stage s takes the R_s points at stride M / R_s of each
// block of M points (M = n, n / R_1, ...), transforms them in registers and
// writes them back where they were, times W_M^(j k).  Frequency
// k = k_1 + R_1 (k_2 + R_2 (...)) ends at position (... (k_1) R_2 + k_2) R_3
// + ...; the inverse runs the stages backwards from there.  Nothing is
// reordered in between: the diffusion factors are tabulated by position, and
// position 0 is frequency 0.  In-place stages need one buffer, so a whole
// z plane (up to ~28000 FP32 points) fits one block and
//   k_mx_xy : Yi, X and the next step's Yf in one trip of a plane, and
//   k_mx_s  : the z pass (and, where a plane does not fit or there are too
//             few planes for the SMs, the separate y passes)
// make a double step two launches.  Radices up to 16 are compile-time
// butterflies chosen by a switch that is uniform over the block.
//
// Bound: FP32 the latency of the stages (a barrier each) and of the launches,
// FP64 the FP64 pipe: one warp instruction per 64 cycles on each SM quarter,
// so FP64 plans with fewer points than lanes take small radices, which leave
// every quarter a short program.
#pragma once
#include "bulk_tma.cuh"

namespace mxk {

constexpr int kMaxStages = 6;
struct Axis {
  int n, nst, tw_off;
  int rad[kMaxStages];
  int m[kMaxStages];            // block length M of the stage
  unsigned mg[kMaxStages];      // 2^20 / (M / R) + 1: division by M / R of u < n <= 1024
};

template <typename T>
struct Dev {
  int gx, gy, gz;
  Axis ax, ay, az;
  const cplx<T>* tw;            // twiddle tables (offsets in the axes)
  const T* fk;                  // by position: g_xy hi, lo [gy gx] each, g_z / N hi, lo [gz] each
  const BulkDev<T>* I;
  cplx<T>* spec;
  cplx<T>* slices;
  const T* E;
  float2* dcin;                 // [gz] FP32 (0, 0) pencil before the z pass, kept by the pass before it
  float2* dcout;                // [gz] the pencil convolved by the z pass
  const float2* dcc;            // [gz] its kernel, (hi, lo)
  int pitch;                    // row pitch of a plane in shared memory (odd)
  unsigned mgx, mgj;            // divisions by gx, and by gx over the first x radix (div_magic)
};

__host__ __device__ __forceinline__ unsigned div_magic(int d) {
  return d <= 1 ? 0u : 0xffffffffu / (unsigned)d + 1;   // ceil(2^32 / d)
}
// t / d for t d < 2^32
__device__ __forceinline__ int fdiv(int t, unsigned mg) { return mg ? (int)__umulhi((unsigned)t, mg) : t; }

// W_R^m of the composite butterflies below (m = n1 k2), W = c - i sg s
template <int R>
__device__ __forceinline__ void wr(int m, double& c, double& s) {
  constexpr double c6[3] = {1.0, 0.5, -0.5}, s6[3] = {0.0, K_SQRT3_2, K_SQRT3_2};
  constexpr double c9[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405};
  constexpr double s9[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937, K_SQRT3_2, 0.34202014332566873304};
  constexpr double c10[5] = {1.0, -K_C5_2, K_C5_1, -K_C5_1, K_C5_2};
  constexpr double s10[5] = {0.0, K_S5_2, K_S5_1, K_S5_1, K_S5_2};
  constexpr double c15[9] = {1.0, 0.91354545764260089550, 0.66913060635885821383, K_C5_1, -0.10452846326765347140,
                             -0.5, K_C5_2, -0.97814760073380563793, -0.97814760073380563793};
  constexpr double s15[9] = {0.0, 0.40673664307580020775, 0.74314482547739423501, K_S5_1, 0.99452189536827333692,
                             K_SQRT3_2, K_S5_2, 0.20791169081775933710, -0.20791169081775933710};
  if constexpr (R == 6) { c = c6[m]; s = s6[m]; }
  else if constexpr (R == 9) { c = c9[m]; s = s9[m]; }
  else if constexpr (R == 10) { c = c10[m]; s = s10[m]; }
  else { c = c15[m]; s = s15[m]; }
}

template <typename T, int R>
__device__ __forceinline__ void dft(cplx<T>* v, int sg);

// R = P Q, natural order in and out (as dft_pq)
template <typename T, int P, int Q>
__device__ __forceinline__ void dft_comp(cplx<T>* v, int sg) {
  cplx<T> a[P][Q];
#pragma unroll
  for (int n1 = 0; n1 < P; ++n1) {
    cplx<T> t[Q];
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) t[n2] = v[n1 + P * n2];
    dft<T, Q>(t, sg);
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2) {
      if (n1 * k2 == 0) { a[n1][k2] = t[k2]; continue; }
      double c, s;
      wr<P * Q>(n1 * k2, c, s);
      a[n1][k2] = mk<T>(t[k2].x * (T)c + sg * t[k2].y * (T)s, t[k2].y * (T)c - sg * t[k2].x * (T)s);
    }
  }
#pragma unroll
  for (int k2 = 0; k2 < Q; ++k2) {
    cplx<T> t[P];
#pragma unroll
    for (int n1 = 0; n1 < P; ++n1) t[n1] = a[n1][k2];
    dft<T, P>(t, sg);
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) v[k2 + Q * k1] = t[k1];
  }
}

template <typename T, int R>
__device__ __forceinline__ void dft(cplx<T>* v, int sg) {
  if constexpr (R == 6) dft_comp<T, 2, 3>(v, sg);
  else if constexpr (R == 9) dft_comp<T, 3, 3>(v, sg);
  else if constexpr (R == 10) dft_comp<T, 2, 5>(v, sg);
  else if constexpr (R == 15) dft_comp<T, 3, 5>(v, sg);
  else dft_c<T, R>(v, sg);
}

// One stage over `lines` lines at pitch ls (point pitch es), twiddle table
// W_n at element `tw` of shared memory: forward (SG = 1) transforms, then
// multiplies by W_M^(j k); inverse (SG = -1) multiplies by the conjugate, then
// transforms.  The points are read at element `buf` of shared memory and
// written back there, except that SRC_G reads them from, and DST_G writes
// them to, global memory (gp, pitches gls and ges); dc: FP32 value that
// replaces point 0 of line 0 on the way in (SRC_G) or receives it (DST_G).
struct Geo {
  int n, R, M;
  unsigned mg;
  int lines;
  unsigned mgl;
  int ls, es;
};
template <typename T>
struct Glob {
  cplx<T>* p;
  int ls, es;
  float2* dc;
};
enum { IO_SMEM = 0, SRC_G = 1, DST_G = 2 };

template <typename T, int SG, int R, int IO>
__device__ __forceinline__ void stage_r(int buf, int tw, const Geo& g, const Glob<T>& G) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
  const int Mp = g.M / R, tws = g.n / g.M;
  const int total = g.n / R * g.lines;
  const int st = Mp * g.es;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int u = fdiv(t, g.mgl), l = t - u * g.lines;
    const int b = (int)(((unsigned)u * g.mg) >> 20), j = u - b * Mp;
    const int at = b * g.M + j;
    cplx<T>* p = sm + buf + l * g.ls + at * g.es;
    cplx<T> v[R];
    if constexpr (IO == SRC_G) {
      const cplx<T>* q = G.p + (size_t)l * G.ls + (size_t)at * G.es;
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = q[(size_t)(r * Mp) * G.es];
      if constexpr (sizeof(T) == 4)
        if (t == 0 && G.dc) v[0] = *G.dc;
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * st];
    }
    const cplx<T>* w = sm + tw;
    const int ji = j * tws;
    if (SG < 0 && j) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmulc<T>(v[r], w[ji * r]);
    }
    dft<T, R>(v, SG);
    if (SG > 0 && j) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul<T>(v[r], w[ji * r]);
    }
    if constexpr (IO == DST_G) {
      cplx<T>* q = G.p + (size_t)l * G.ls + (size_t)at * G.es;
#pragma unroll
      for (int r = 0; r < R; ++r) q[(size_t)(r * Mp) * G.es] = v[r];
      if constexpr (sizeof(T) == 4)
        if (t == 0 && G.dc) *G.dc = v[0];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) p[r * st] = v[r];
    }
  }
}

#define ADSCF_MX_SWITCH(R_, CALL)                                                        \
  switch (R_) {                                                                          \
    case 2: CALL(2); break;                                                              \
    case 3: CALL(3); break;                                                              \
    case 4: CALL(4); break;                                                              \
    case 5: CALL(5); break;                                                              \
    case 6: CALL(6); break;                                                              \
    case 8: CALL(8); break;                                                              \
    case 9: CALL(9); break;                                                              \
    case 10: CALL(10); break;                                                            \
    case 12: CALL(12); break;                                                            \
    case 15: CALL(15); break;                                                            \
    default: CALL(16); break;                                                            \
  }

template <typename T, int SG>
__device__ __noinline__ void stage(int buf, int tw, Geo g) {
  const Glob<T> none{};
#define ADSCF_MX_CALL(R_) stage_r<T, SG, R_, IO_SMEM>(buf, tw, g, none)
  ADSCF_MX_SWITCH(g.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
}
template <typename T, int SG, int IO>
__device__ __noinline__ void stage_io(int buf, int tw, Geo g, Glob<T> G) {
#define ADSCF_MX_CALL(R_) stage_r<T, SG, R_, IO>(buf, tw, g, G)
  ADSCF_MX_SWITCH(g.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
}

__device__ __forceinline__ Geo geo(const Axis& A, int s, int lines, unsigned mgl, int ls, int es) {
  return Geo{A.n, A.rad[s], A.m[s], A.mg[s], lines, mgl, ls, es};
}
// stages [s0, s1) of the lines in shared memory, a barrier after each; the
// inverse runs them from s1 - 1 down
template <typename T, int SG>
__device__ __forceinline__ void stages(int buf, int tw, const Axis& A, int s0, int s1, int lines, unsigned mgl,
                                       int ls, int es) {
  for (int i = s0; i < s1; ++i) {
    stage<T, SG>(buf, tw, geo(A, SG > 0 ? i : s1 - 1 - (i - s0), lines, mgl, ls, es));
    __syncthreads();
  }
}

// Last forward stage, diffusion factor and first inverse stage of the z lines
// in one visit of the points (both stages have M = R, no twiddles).  fz: the
// g_z / N factors by position at byte offset of shared memory (hi [n], lo
// [n]); fxy: the columns' g_xy (hi, with lo at + nxy).
template <typename T, int R>
__device__ __forceinline__ void mid_r(int buf, const Geo& g, int fz_off, const T* fxy, int nxy) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
  const T* fz = reinterpret_cast<const T*>(smraw + fz_off);
  const int total = g.n / R * g.lines;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int u = fdiv(t, g.mgl), l = t - u * g.lines;
    cplx<T>* p = sm + buf + l * g.ls + u * R * g.es;
    const T ah = __ldg(fxy + l);
    T al = (T)0;
    if constexpr (sizeof(T) == 4) al = __ldg(fxy + nxy + l);
    cplx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[r * g.es];
    if constexpr (R > 1) dft<T, R>(v, +1);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const T bh = fz[u * R + r];
      if constexpr (sizeof(T) == 4) {   // compensated product, one rounding
        const float bl = fz[g.n + u * R + r];
        const float gh = ah * bh;
        const float gl = fmaf(ah, bh, -gh) + fmaf(ah, bl, al * bh);
        v[r] = mk<T>(fmaf(v[r].x, gh, v[r].x * gl), fmaf(v[r].y, gh, v[r].y * gl));
      } else {
        const T f = ah * bh;
        v[r] = mk<T>(v[r].x * f, v[r].y * f);
      }
    }
    if constexpr (R > 1) dft<T, R>(v, -1);
#pragma unroll
    for (int r = 0; r < R; ++r) p[r * g.es] = v[r];
  }
}
template <typename T>
__device__ __noinline__ void mid(int buf, Geo g, int fz_off, const T* fxy, int nxy) {
  if (g.R == 1) {
    mid_r<T, 1>(buf, g, fz_off, fxy, nxy);
    return;
  }
#define ADSCF_MX_CALL(R_) mid_r<T, R_>(buf, g, fz_off, fxy, nxy)
  ADSCF_MX_SWITCH(g.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
}

// Last inverse stage of the x rows, node t of both chains and the first
// forward stage in one visit (both stages have M = n: a task holds points
// j + r n / R of a row; tasks of a row are neighbours, so the Boltzmann
// factors and the slice move in runs of n / R points).  E, sl: factors and
// slice at the tile's first point, rows gx apart; f: bits 0-3 = forward /
// backward chain takes the A factor at node t, at node t + 1; bit 4: t <
// Ns, the forward stage follows; init: no inverse, slice = (1, 1).
template <typename T, int R>
__device__ __forceinline__ void real_r(int buf, int tw, const Geo& g, unsigned mgj, const T* E, cplx<T>* sl,
                                       unsigned f, bool init) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
  const int Mp = g.n / R;
  const int total = Mp * g.lines;
  const bool fA = f & 1, bA = f & 2, fA2 = f & 4, bA2 = f & 8, more = f & 16;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int l = fdiv(t, mgj), j = t - l * Mp;
    cplx<T>* p = sm + buf + l * g.ls + j;
    const size_t gp = (size_t)l * g.n + j;
    const cplx<T>* w = sm + tw;
    cplx<T> v[R];
    if (!init) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * Mp];
      if constexpr (R > 1) {
        if (j) {
#pragma unroll
          for (int r = 1; r < R; ++r) v[r] = cmulc<T>(v[r], w[j * r]);
        }
        dft<T, R>(v, -1);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const EPt<T> ev = load_ept(E, gp + (size_t)r * Mp);
      if (init) {
        v[r] = mk<T>(fA ? ev.a : ev.b, bA ? ev.a : ev.b);
        sl[gp + (size_t)r * Mp] = mk<T>((T)1, (T)1);
      } else {
        const cplx<T> q = mk<T>(emul(v[r].x, fA ? ev.a : ev.b, fA ? ev.al : ev.bl),
                                emul(v[r].y, bA ? ev.a : ev.b, bA ? ev.al : ev.bl));
        sl[gp + (size_t)r * Mp] = q;
        v[r] = mk<T>(emul(q.x, fA2 ? ev.a : ev.b, fA2 ? ev.al : ev.bl),
                     emul(q.y, bA2 ? ev.a : ev.b, bA2 ? ev.al : ev.bl));
      }
    }
    if (!more) continue;
    if constexpr (R > 1) {
      dft<T, R>(v, +1);
      if (j) {
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul<T>(v[r], w[j * r]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) p[r * Mp] = v[r];
  }
}
template <typename T>
__device__ __noinline__ void real_mid(int buf, int tw, Geo g, unsigned mgj, const T* E, cplx<T>* sl, unsigned f,
                                      bool init) {
  if (g.R == 1) {
    real_r<T, 1>(buf, tw, g, mgj, E, sl, f, init);
    return;
  }
#define ADSCF_MX_CALL(R_) real_r<T, R_>(buf, tw, g, mgj, E, sl, f, init)
  ADSCF_MX_SWITCH(g.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
}

template <typename T>
__device__ __forceinline__ void load_tw(cplx<T>* dst, const Dev<T>& D, const Axis& A) {
  for (int i = threadIdx.x; i < A.n; i += blockDim.x) dst[i] = D.tw[A.tw_off + i];
}

}  // namespace mxk

// ---------------------------------------------------------------------------
// Real-space pass of `rows` x-rows per block: [inverse y,] inverse x, node t
// of both chains (slice store), times E(t + 1), forward x [, forward y].
// PLANES: the rows are one z plane (rows = gy > 1, blockIdx.x = z) and the y
// transforms belong to the pass; their outermost stages read and write the
// spectrum directly.  Otherwise rows [blockIdx.x rows, + rows) of the grid, x
// only.  t = 0 starts the chains: slice 0 = (1, 1).
// Where the block handles whole (0, 0) pencil entries -- planes, or every row
// of a one-point y axis -- it takes their values of the z pass from D.dcout
// and leaves those for the next one in D.dcin (FP32).
// Shared memory: rows pitch + gx + (PLANES ? gy : 0) points.
// ---------------------------------------------------------------------------
template <typename T, bool PLANES>
__global__ void __launch_bounds__(512)
k_mx_xy(const __grid_constant__ mxk::Dev<T> D, int t, int rows, unsigned mg_rows) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx<T>* tile = reinterpret_cast<cplx<T>*>(smraw);
  const BulkDev<T>& I = *D.I;
  const int gx = D.gx, pitch = D.pitch;
  const int row0 = blockIdx.x * rows;
  const int nr = PLANES ? rows : min(rows, D.gy * D.gz - row0);
  const unsigned mgl = nr == rows ? mg_rows : mxk::div_magic(nr);
  const int ne = nr * gx;
  const int o_twx = rows * pitch, o_twy = o_twx + gx;
  const size_t base = (size_t)row0 * gx;
  const int ns = I.ns;
  tmak::pdl_launch_dependents();
  mxk::load_tw<T>(tile + o_twx, D, D.ax);
  if constexpr (PLANES) mxk::load_tw<T>(tile + o_twy, D, D.ay);
  const int tt = t == 0 ? 1 : t;
  const bool more = t == 0 || t < ns;
  const unsigned f = (chain_type_fwd(I, tt) == 0 ? 1u : 0u) | (chain_type_bwd(I, tt) == 0 ? 2u : 0u) |
                     (chain_type_fwd(I, t + 1) == 0 ? 4u : 0u) | (chain_type_bwd(I, t + 1) == 0 ? 8u : 0u) |
                     (more ? 16u : 0u);
  const bool dcrow = sizeof(T) == 4 && (PLANES || D.gy == 1);
  cplx<T>* sl = D.slices + (size_t)t * (size_t)I.npts + base;
  const T* E = D.E + base * (sizeof(T) == 4 ? 4 : 2);
  const int nx = D.ax.nst, ny = D.ay.nst;
  tmak::pdl_wait();
  if constexpr (PLANES) __syncthreads();   // twiddles
  if (t > 0) {
    {  // the tile's Boltzmann factors on their way to L1 while it is transformed
      const char* e0 = reinterpret_cast<const char*>(E);
      for (int i = threadIdx.x * 128; i < ne * 16; i += blockDim.x * 128) tmak::prefetch_l1(e0 + i);
    }
    if constexpr (PLANES) {
      const mxk::Glob<T> G{D.spec + base, 1, gx, dcrow ? D.dcout + blockIdx.x : nullptr};
      mxk::stage_io<T, -1, mxk::SRC_G>(0, o_twy, mxk::geo(D.ay, ny - 1, gx, D.mgx, 1, pitch), G);
      __syncthreads();
      mxk::stages<T, -1>(0, o_twy, D.ay, 0, ny - 1, gx, D.mgx, 1, pitch);
    } else {
#pragma unroll 4
      for (int e = threadIdx.x; e < ne; e += blockDim.x) {
        const int r = mxk::fdiv(e, D.mgx), x = e - r * gx;
        tile[r * pitch + x] = D.spec[base + e];
      }
      if constexpr (sizeof(T) == 4) {
        if (dcrow) {
          __syncthreads();
          for (int r = threadIdx.x; r < nr; r += blockDim.x) tile[r * pitch] = D.dcout[row0 + r];
        }
      }
      __syncthreads();
    }
    mxk::stages<T, -1>(0, o_twx, D.ax, 1, nx, nr, mgl, pitch, 1);
  } else if constexpr (!PLANES) {
    __syncthreads();   // twiddles
  }
  {
    mxk::Geo g = nx ? mxk::geo(D.ax, 0, nr, mgl, pitch, 1) : mxk::Geo{1, 1, 1, 0u, nr, mgl, pitch, 1};
    mxk::real_mid<T>(0, o_twx, g, D.mgj, E, sl, f, t == 0);
  }
  if (!more) return;
  __syncthreads();
  mxk::stages<T, +1>(0, o_twx, D.ax, 1, nx, nr, mgl, pitch, 1);
  if constexpr (PLANES) {
    mxk::stages<T, +1>(0, o_twy, D.ay, 0, ny - 1, gx, D.mgx, 1, pitch);
    const mxk::Glob<T> G{D.spec + base, 1, gx, dcrow ? D.dcin + blockIdx.x : nullptr};
    mxk::stage_io<T, +1, mxk::DST_G>(0, o_twy, mxk::geo(D.ay, ny - 1, gx, D.mgx, 1, pitch), G);
  } else {
#pragma unroll 4
    for (int e = threadIdx.x; e < ne; e += blockDim.x) {
      const int r = mxk::fdiv(e, D.mgx), x = e - r * gx;
      D.spec[base + e] = tile[r * pitch + x];
    }
    if constexpr (sizeof(T) == 4) {
      if (dcrow)
        for (int r = threadIdx.x; r < nr; r += blockDim.x) D.dcin[row0 + r] = tile[r * pitch];
    }
  }
}

// ---------------------------------------------------------------------------
// Strided passes: tiles of `cols` (a power of two) neighbouring columns.
// KIND 0 forward y, 1 inverse y (columns x of plane z, tiles do not cross
// planes), 2 z (columns (y, x)).  The outermost stages read and write the
// spectrum directly.  The z pass has `ntiles` blocks of columns, then blocks
// whose warps convolve the FP32 (0, 0) pencil, one output per warp, from
// D.dcin into D.dcout (the columns' own result for it is replaced by the next
// pass).  The y passes keep and replace the pencil's entries.
// Shared memory: n cols + n points, and 2 n factors (z).
// ---------------------------------------------------------------------------
template <typename T, int KIND>
__global__ void __launch_bounds__(256)
k_mx_s(const __grid_constant__ mxk::Dev<T> D, int cols, int ntiles) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx<T>* tile = reinterpret_cast<cplx<T>*>(smraw);
  constexpr bool zdir = KIND == 2;
  const mxk::Axis& A = zdir ? D.az : D.ay;
  const int n = A.n, gx = D.gx, nxy = gx * D.gy, ns = A.nst;
  tmak::pdl_launch_dependents();
  if constexpr (zdir && sizeof(T) == 4) {
    if ((int)blockIdx.x >= ntiles) {
      float2* in = reinterpret_cast<float2*>(smraw);
      float2* c = in + n;
      for (int i = threadIdx.x; i < n; i += blockDim.x) c[i] = D.dcc[i];
      tmak::pdl_wait();
      for (int i = threadIdx.x; i < n; i += blockDim.x) in[i] = D.dcin[i];
      __syncthreads();
      const int nw = blockDim.x >> 5;
      const int z = ((int)blockIdx.x - ntiles) * nw + (threadIdx.x >> 5);
      if (z < n) {
        const float2 o = tmak::dc_point(in, c, n, z);
        if ((threadIdx.x & 31) == 0) D.dcout[z] = o;
      }
      return;
    }
  }
  const int o_tw = n * cols;
  const int fz_off = (o_tw + n) * (int)sizeof(cplx<T>);
  mxk::load_tw<T>(tile + o_tw, D, A);
  if constexpr (zdir) {
    T* fz = reinterpret_cast<T*>(smraw + fz_off);
    const T* gzt = D.fk + 2 * (size_t)nxy;
    for (int i = threadIdx.x; i < 2 * n; i += blockDim.x) fz[i] = gzt[i];
  }
  const int lc = __ffs(cols) - 1;
  size_t base;
  int nl, es;
  int z = 0, x0 = 0;
  if constexpr (zdir) {
    const int L0 = blockIdx.x * cols;
    base = L0;
    nl = min(cols, nxy - L0);
    es = nxy;
  } else {
    const int tpp = (gx + cols - 1) >> lc;
    z = blockIdx.x / tpp;
    x0 = (blockIdx.x - z * tpp) << lc;
    base = (size_t)z * nxy + x0;
    nl = min(cols, gx - x0);
    es = gx;
  }
  const unsigned mgl = nl == cols ? (lc ? 1u << (32 - lc) : 0u) : mxk::div_magic(nl);
  const bool dcl = sizeof(T) == 4 && !zdir && x0 == 0;
  const mxk::Glob<T> in{D.spec + base, 1, es, dcl && KIND == 1 ? D.dcout + z : nullptr};
  const mxk::Glob<T> out{D.spec + base, 1, es, dcl && KIND == 0 ? D.dcin + z : nullptr};
  tmak::pdl_wait();
  __syncthreads();
  if constexpr (KIND < 2) {
    constexpr int SG = KIND == 0 ? +1 : -1;
    const int first = SG > 0 ? 0 : ns - 1, last = SG > 0 ? ns - 1 : 0;
    if (ns == 1) {   // one stage: through shared memory, then out
      mxk::stage_io<T, SG, mxk::SRC_G>(0, o_tw, mxk::geo(A, 0, nl, mgl, 1, cols), in);
      __syncthreads();
      for (int e = threadIdx.x; e < n << lc; e += blockDim.x) {
        const int j = e >> lc, c = e & (cols - 1);
        if (c < nl) D.spec[base + (size_t)j * es + c] = tile[e];
      }
      if constexpr (sizeof(T) == 4 && KIND == 0) {
        if (dcl && threadIdx.x == 0) D.dcin[z] = tile[0];
      }
      return;
    }
    mxk::stage_io<T, SG, mxk::SRC_G>(0, o_tw, mxk::geo(A, first, nl, mgl, 1, cols), in);
    __syncthreads();
    mxk::stages<T, SG>(0, o_tw, A, 1, ns - 1, nl, mgl, 1, cols);
    mxk::stage_io<T, SG, mxk::DST_G>(0, o_tw, mxk::geo(A, last, nl, mgl, 1, cols), out);
  } else {
    if (ns < 2) {   // the middle visit only: through shared memory
      for (int e = threadIdx.x; e < n << lc; e += blockDim.x) {
        const int j = e >> lc, c = e & (cols - 1);
        if (c < nl) tile[e] = D.spec[base + (size_t)j * es + c];
      }
      __syncthreads();
    } else {
      mxk::stage_io<T, +1, mxk::SRC_G>(0, o_tw, mxk::geo(A, 0, nl, mgl, 1, cols), in);
      __syncthreads();
      mxk::stages<T, +1>(0, o_tw, A, 1, ns - 1, nl, mgl, 1, cols);
    }
    const int R = ns ? A.rad[ns - 1] : 1;
    mxk::mid<T>(0, mxk::Geo{n, R, R, 0u, nl, mgl, 1, cols}, fz_off, D.fk + base, nxy);
    __syncthreads();
    if (ns < 2) {
      for (int e = threadIdx.x; e < n << lc; e += blockDim.x) {
        const int j = e >> lc, c = e & (cols - 1);
        if (c < nl) D.spec[base + (size_t)j * es + c] = tile[e];
      }
    } else {
      mxk::stages<T, -1>(0, o_tw, A, 1, ns - 1, nl, mgl, 1, cols);
      mxk::stage_io<T, -1, mxk::DST_G>(0, o_tw, mxk::geo(A, 0, nl, mgl, 1, cols), out);
    }
  }
}

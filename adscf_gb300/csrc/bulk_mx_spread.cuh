// bulk_mx_spread.cuh -- the mixed-radix passes of bulk_mx.cuh with one output of
// a butterfly per lane, for FP64 grids with fewer points than the GPU has FP64
// lanes.
//
// An FP64 warp instruction holds its SM quarter for 64 cycles whatever its
// lanes do, so a grid too small to give every quarter a warp of butterflies
// pays for the length of one lane's program: 28 FP64 instructions a radix-4
// stage with its twiddles.  Here the R lanes of a butterfly read its R points
// and compute one output each (10 instructions for radix 4, 6, 12 and 20 for
// 2, 3 and 5), on R times as many warps.  Radices are 2 to 5.
//
// Stages are those of bulk_mx.cuh, in place, but an inverse stage finds its
// points already multiplied by its twiddles: each inverse stage multiplies
// its outputs (one product a lane) for the next one of the axis, across the y
// cut too.  The spectrum between the passes therefore differs from the other
// kernels' by those factors, and a run uses one family.
//
// Measured (us a double step, against a butterfly per lane): see mx_setup.
#pragma once
#include "bulk_mx.cuh"

namespace mxk {

static __constant__ double kCos5[5] = {1.0, 0.30901699437494742410, -0.80901699437494742410, -0.80901699437494742410,
                                       0.30901699437494742410};
static __constant__ double kSin5[5] = {0.0, 0.95105651629515357212, 0.58778525229247312917, -0.58778525229247312917,
                                       -0.95105651629515357212};

__device__ __forceinline__ double flip(double x, unsigned s) {   // s: 0 or the sign bit
  return __hiloint2double(__double2hiint(x) ^ (int)s, __double2loint(x));
}

// output k of the R-point transform of x (SG: 1 forward, -1 inverse)
template <int R, int SG>
__device__ __forceinline__ double2 dft_out(const double2 (&x)[R], int k) {
  if constexpr (R == 2) {
    const unsigned s = (unsigned)k << 31;
    return make_double2(x[0].x + flip(x[1].x, s), x[0].y + flip(x[1].y, s));
  } else if constexpr (R == 4) {
    const unsigned s = (unsigned)(k & 1) << 31;
    const double2 p = make_double2(x[0].x + flip(x[2].x, s), x[0].y + flip(x[2].y, s));
    const double2 q = make_double2(x[1].x + flip(x[3].x, s), x[1].y + flip(x[3].y, s));
    // q times (-i SG)^k
    const bool odd = k & 1;
    const unsigned m = odd ? ((k == 1) == (SG > 0) ? 0u : 0x80000000u) : (unsigned)(k >> 1) << 31;
    const double re = odd ? q.y : q.x, im = odd ? q.x : q.y;
    return make_double2(p.x + flip(re, m), p.y + flip(im, odd ? m ^ 0x80000000u : m));
  } else if constexpr (R == 3) {
    const double c = k ? -0.5 : 1.0;
    const double s = k == 0 ? 0.0 : (k == 1) == (SG > 0) ? K_SQRT3_2 : -K_SQRT3_2;
    const double2 a = make_double2(x[1].x + x[2].x, x[1].y + x[2].y), d = make_double2(x[1].x - x[2].x, x[1].y - x[2].y);
    return make_double2(fma(s, d.y, fma(c, a.x, x[0].x)), fma(-s, d.x, fma(c, a.y, x[0].y)));
  } else {
    static_assert(R == 5, "radix");
    const int k2 = k < 3 ? 2 * k : 2 * k - 5;
    const double c1 = kCos5[k], c2 = kCos5[k2], s1 = SG * kSin5[k], s2 = SG * kSin5[k2];
    const double2 a = make_double2(x[1].x + x[4].x, x[1].y + x[4].y), d = make_double2(x[1].x - x[4].x, x[1].y - x[4].y);
    const double2 b = make_double2(x[2].x + x[3].x, x[2].y + x[3].y), e = make_double2(x[2].x - x[3].x, x[2].y - x[3].y);
    return make_double2(fma(s2, e.y, fma(s1, d.y, fma(c2, b.x, fma(c1, a.x, x[0].x)))),
                        fma(-s2, e.x, fma(-s1, d.x, fma(c2, b.y, fma(c1, a.y, x[0].y)))));
  }
}

#define ADSCF_MXS_SWITCH(R_, CALL) \
  switch (R_) {                    \
    case 2: CALL(2); break;        \
    case 3: CALL(3); break;        \
    case 4: CALL(4); break;        \
    default: CALL(5); break;       \
  }

// A warp takes 32 / R butterflies at a time: lane i output i / (32 / R) of
// butterfly i % (32 / R).
template <int R>
struct Lane {
  static constexpr int G = 32 / R;
  int first, step, i, k;
  bool in;
  __device__ __forceinline__ Lane() {
    const int lane = threadIdx.x & 31;
    i = lane % G;
    k = lane / G;
    in = k < R;
    first = (threadIdx.x >> 5) * G;
    step = (blockDim.x >> 5) * G;
  }
};

// One stage (as stage_r); V: the stage before, b0: blocks of the axis before the tile's first one,
// in stages of S's length per row block
template <int SG, bool SRC, int R>
__device__ __forceinline__ void spread_r(const Step& S, const Prev& V, double2* sm, int tile_j, int b0, double2* g, int nl) {
  const Lane<R> ln;
  const double2* w = sm + S.tw;
  for (int t0 = ln.first; t0 < S.total; t0 += ln.step) {
    const int t = t0 + ln.i;
    const bool live = ln.in && t < S.total;
    double2 o = make_double2(0.0, 0.0);
    double2 *p = nullptr, *q = nullptr;
    int lo = 0;
    if (live) {
      const int u = fdiv(t, S.mgl), l = t - u * S.lines;
      const int b = (int)(((unsigned)u * S.mg) >> 20), j = u - b * S.mp;
      const int at = b * S.m + j, hi = l >> S.lsh;
      lo = l & S.lmask;
      p = sm + lo * S.ls + hi * S.ls2 + at * S.es;
      q = g ? g + (size_t)lo * S.gls + (size_t)hi * S.gls2 + (size_t)at * S.ges : nullptr;
      const int st = S.mp * S.es;
      const size_t gst = (size_t)S.mp * S.ges;
      double2 v[R];
      if (SRC && g) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = lo < nl ? q[r * gst] : make_double2(0.0, 0.0);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = p[r * st];
      }
      int wi;
      if (SG > 0) wi = (S.jmul * j + S.jin * tile_j) * S.tws * ln.k;
      else wi = V.rp ? (S.jmul * (j + ln.k * S.mp) + S.jin * tile_j) * ((b + b0 * V.nb) % V.rp) * V.twp : 0;
      const double2 wv = w[wi];
      o = dft_out<R, SG>(v, ln.k);
      if (wi) o = SG > 0 ? cmul<double>(o, wv) : cmulc<double>(o, wv);
      p += ln.k * st;
      if (!SRC && g) q += ln.k * gst;
    }
    __syncwarp();
    if (live) {
      if (!SRC && g) {
        if (lo < nl) *q = o;
      } else {
        *p = o;
      }
    }
  }
}

// the z lines' last forward stage, diffusion factor and first inverse stage
// (as mid_r); rp, twp: radix and twiddle step of the stage before, w: z twiddles
template <int R, int MODE>
__device__ __forceinline__ void spread_mid_r(const Dev<double>& D, double2* sm, const double* fz, const double* fxy,
                                             int nl, int rp, int twp, const double2* w, const Side<double>& sd) {
  const Lane<R> ln;
  const int lines = D.mi << D.lc, total = D.gz / R * lines;
  for (int t0 = ln.first; t0 < total; t0 += ln.step) {
    const int t = t0 + ln.i;
    const int u = fdiv(t, D.mgz), l = t - u * lines;
    const int c = l & (D.cols - 1), yy = l >> D.lc;
    const bool live = ln.in && t < total && c < nl;
    double2* p = sm + yy * D.pb + ((u * R) << D.lc) + c;
    double2 o;
    if (live) {
      const double f = __ldg(fxy + (size_t)yy * D.gx + c) * fz[u * R + ln.k];
      double2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r << D.lc];
      o = dft_out<R, 1>(v, ln.k);
      if constexpr (MODE != kPlain) sd.keep[(size_t)(((u * R + ln.k) * D.mi + yy) << D.lc) + c] = o;
      o = make_double2(o.x * f, o.y * f);
    }
    if constexpr (MODE == kSpec) continue;
    __syncwarp();
    if (live) p[ln.k << D.lc] = o;
    __syncwarp();
    if (live) {
      double2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r << D.lc];
      o = dft_out<R, -1>(v, ln.k);
      const int wi = rp ? ln.k * (u % rp) * twp : 0;
      if (wi) o = cmulc<double>(o, w[wi]);
    }
    __syncwarp();
    if (live) p[ln.k << D.lc] = o;
  }
}

// the x rows' last inverse stage, node t and first forward stage (as real_r)
template <int R, bool FROM>
__device__ __forceinline__ void spread_real_r(const Dev<double>& D, double2* sm, const double* E, double2* sl, unsigned f,
                                              bool init) {
  const Lane<R> ln;
  const int Mp = D.gx / R, total = Mp * D.ro;
  const size_t rs = (size_t)D.mi * D.gx;
  const bool fA = f & 1, bA = f & 2, fA2 = f & 4, bA2 = f & 8, more = f & 16;
  const double2* w = sm + D.ro * D.pitch;
  for (int t0 = ln.first; t0 < total; t0 += ln.step) {
    const int t = t0 + ln.i;
    const bool live = ln.in && t < total;
    const int l = fdiv(t, D.mgj), j = t - l * Mp;
    double2* p = sm + l * D.pitch + j;
    double2 o;
    if (live) {
      const size_t g = l * rs + j + ln.k * Mp;
      const EPt<double> ev = load_ept(E, g);
      if constexpr (FROM) {
        const double2 q = sl[g];
        o = make_double2(q.x * (fA2 ? ev.a : ev.b), q.y * (bA2 ? ev.a : ev.b));
      } else if (init) {
        sl[g] = make_double2(1.0, 1.0);
        o = make_double2(fA ? ev.a : ev.b, bA ? ev.a : ev.b);
      } else {
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = p[r * Mp];
        const double2 q0 = dft_out<R, -1>(v, ln.k);
        const double2 q = make_double2(q0.x * (fA ? ev.a : ev.b), q0.y * (bA ? ev.a : ev.b));
        sl[g] = q;
        o = make_double2(q.x * (fA2 ? ev.a : ev.b), q.y * (bA2 ? ev.a : ev.b));
      }
    }
    if (!more) continue;
    __syncwarp();
    if (live) p[ln.k * Mp] = o;
    __syncwarp();
    if (live) {
      double2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * Mp];
      o = dft_out<R, 1>(v, ln.k);
      if (j && ln.k) o = cmul<double>(o, w[j * ln.k]);
    }
    __syncwarp();
    if (live) p[ln.k * Mp] = o;
  }
}

// a one-point x axis: node t of row l in lane l
template <bool FROM>
__device__ __forceinline__ void spread_real_1(const Dev<double>& D, double2* sm, const double* E, double2* sl, unsigned f,
                                              bool init) {
  const size_t rs = (size_t)D.mi * D.gx;
  const bool fA = f & 1, bA = f & 2, fA2 = f & 4, bA2 = f & 8;
  for (int l = threadIdx.x; l < D.ro; l += blockDim.x) {
    double2* p = sm + l * D.pitch;
    const EPt<double> ev = load_ept(E, l * rs);
    if constexpr (FROM) {
      const double2 q = sl[l * rs];
      *p = make_double2(q.x * (fA2 ? ev.a : ev.b), q.y * (bA2 ? ev.a : ev.b));
      continue;
    }
    double2 q = make_double2(1.0, 1.0);
    if (!init) q = make_double2(p->x * (fA ? ev.a : ev.b), p->y * (bA ? ev.a : ev.b));
    sl[l * rs] = q;
    if (init) *p = make_double2(fA ? ev.a : ev.b, bA ? ev.a : ev.b);
    else *p = make_double2(q.x * (fA2 ? ev.a : ev.b), q.y * (bA2 ? ev.a : ev.b));
  }
}

}  // namespace mxk

// k_mx_a
template <bool FROM>
__device__ __forceinline__ void spread_a_body(const mxk::Dev<double>& D, const mxk::Spread& W, int t) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sm = reinterpret_cast<double2*>(smraw);
  const BulkDev<double>& I = *D.io.I;
  const int gx = D.gx, ro = D.ro, mi = D.mi;
  const int z = blockIdx.x / mi, j = blockIdx.x - z * mi;
  const size_t base = ((size_t)z * D.gy + j) * gx;
  const int ns = I.ns;
  tmak::pdl_launch_dependents();
  {
    double2* tw = sm + ro * D.pitch;
    for (int i = threadIdx.x; i < gx; i += blockDim.x) tw[i] = D.tw[D.tw_x + i];
    if (ro > 1)
      for (int i = threadIdx.x; i < D.gy; i += blockDim.x) tw[gx + i] = D.tw[D.tw_y + i];
  }
  const int tt = t == 0 ? 1 : t;
  const bool more = t == 0 || t < ns;
  const unsigned f = (chain_type_fwd(I, tt) == 0 ? 1u : 0u) | (chain_type_bwd(I, tt) == 0 ? 2u : 0u) |
                     (chain_type_fwd(I, t + 1) == 0 ? 4u : 0u) | (chain_type_bwd(I, t + 1) == 0 ? 8u : 0u) |
                     (more ? 16u : 0u);
  double2* sl = D.io.slices + (size_t)t * (size_t)I.npts + base;
  const double* E = D.io.E + base * 2;
  double2* g = D.io.spec + base;
  tmak::pdl_wait();
  __syncthreads();
  if (!FROM && t > 0) {
    if (D.a.n == 0) {
      for (int x = threadIdx.x; x < gx; x += blockDim.x) sm[x] = g[x];
      __syncthreads();
    }
    for (int i = D.a.n - 1; i >= 0; --i) {
      const mxk::Step& S = D.a.s[i];
      double2* src = i == D.a.n - 1 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::spread_r<-1, true, R_>(S, W.a[i], sm, j, 0, src, gx)
      ADSCF_MXS_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
      __syncthreads();
    }
  }
  if (D.rx == 1) {
    mxk::spread_real_1<FROM>(D, sm, E, sl, f, t == 0);
  } else {
#define ADSCF_MX_CALL(R_) mxk::spread_real_r<R_, FROM>(D, sm, E, sl, f, t == 0)
    ADSCF_MXS_SWITCH(D.rx, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
  }
  if (!more) return;
  __syncthreads();
  for (int i = 0; i < D.a.n; ++i) {
    const mxk::Step& S = D.a.s[i];
    double2* dst = i == D.a.n - 1 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::spread_r<+1, false, R_>(S, W.a[i], sm, j, 0, dst, gx)
    ADSCF_MXS_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
    if (!dst) __syncthreads();
  }
  if (D.a.n == 0)
    for (int x = threadIdx.x; x < gx; x += blockDim.x) g[x] = sm[x];
}

static __global__ void __launch_bounds__(256, 2)
k_mx_a_spread(const __grid_constant__ mxk::Dev<double> D, const __grid_constant__ mxk::Spread W, int t) {
  spread_a_body<false>(D, W, t);
}
static __global__ void __launch_bounds__(256, 2)
k_mx_a_spread_from(const __grid_constant__ mxk::Dev<double> D, const __grid_constant__ mxk::Spread W, int t) {
  spread_a_body<true>(D, W, t);
}

// k_mx_b
template <int MODE>
__device__ __forceinline__ void spread_b_body(const mxk::Dev<double>& D, const mxk::Spread& W, const mxk::Side<double>& sd) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sm = reinterpret_cast<double2*>(smraw);
  const int gx = D.gx, gz = D.gz, mi = D.mi, nxy = gx * D.gy;
  const int k = blockIdx.x / D.ctiles, c0 = (blockIdx.x - k * D.ctiles) << D.lc;
  const int nl = min(D.cols, gx - c0);
  const int pts = mi * D.pb;
  double* fz = reinterpret_cast<double*>(sm + pts + D.gy + gz);
  tmak::pdl_launch_dependents();
  if (mi > 1)
    for (int i = threadIdx.x; i < D.gy; i += blockDim.x) sm[pts + i] = D.tw[D.tw_y + i];
  for (int i = threadIdx.x; i < gz; i += blockDim.x) sm[pts + D.gy + i] = D.tw[D.tw_z + i];
  for (int i = threadIdx.x; i < gz; i += blockDim.x) fz[i] = D.io.fk[2 * (size_t)nxy + i];
  double2* g = D.io.spec + (size_t)k * mi * gx + c0;
  const double* fxy = D.io.fk + (size_t)k * mi * gx + c0;
  tmak::pdl_wait();
  __syncthreads();
  if (D.b.n == 0) {
    for (int e = threadIdx.x; e < gz << D.lc; e += blockDim.x) {
      const int c = e & (D.cols - 1), zz = e >> D.lc;
      if (c < nl) sm[e] = g[(size_t)zz * nxy + c];
    }
    __syncthreads();
  }
  for (int i = 0; i < D.b.n; ++i) {
    const mxk::Step& S = D.b.s[i];
    double2* src = i == 0 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::spread_r<+1, true, R_>(S, W.b[i], sm, 0, 0, src, nl)
    ADSCF_MXS_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
    __syncthreads();
  }
  if (D.rz == 1) {
    mxk::mid_r<double, 1, MODE>(D, sm, fz, fxy, nl, sd);
  } else {
#define ADSCF_MX_CALL(R_) mxk::spread_mid_r<R_, MODE>(D, sm, fz, fxy, nl, W.zrp, W.ztwp, sm + pts + D.gy, sd)
    ADSCF_MXS_SWITCH(D.rz, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
  }
  if constexpr (MODE == mxk::kSpec) return;
  __syncthreads();
  for (int i = D.b.n - 1; i >= 0; --i) {
    const mxk::Step& S = D.b.s[i];
    double2* dst = i == 0 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::spread_r<-1, false, R_>(S, W.b[i], sm, 0, k, dst, nl)
    ADSCF_MXS_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
    if (!dst) __syncthreads();
  }
  if (D.b.n == 0) {
    for (int e = threadIdx.x; e < gz << D.lc; e += blockDim.x) {
      const int c = e & (D.cols - 1), zz = e >> D.lc;
      if (c < nl) g[(size_t)zz * nxy + c] = sm[e];
    }
  }
}
static __global__ void __launch_bounds__(256, 2)
k_mx_b_spread(const __grid_constant__ mxk::Dev<double> D, const __grid_constant__ mxk::Spread W) {
  spread_b_body<mxk::kPlain>(D, W, mxk::Side<double>{});
}
// with side data of `tile` points a block
template <int MODE>
__global__ void __launch_bounds__(256, 2)
k_mx_b_spread_side(const __grid_constant__ mxk::Dev<double> D, const __grid_constant__ mxk::Spread W, double2* keep, int tile) {
  spread_b_body<MODE>(D, W, mxk::Side<double>{keep + (size_t)blockIdx.x * tile, nullptr});
}

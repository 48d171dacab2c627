// bulk_mx.cuh -- mixed-radix passes of the bulk propagator: grids with a line that
// has no register FFT (lengths of 2, 3 and 5 factors up to 1024), and of the others
// those where they are ahead (create_t in bulk.cu: FP64 but 256^3, FP32 with a line
// of 256 points, and 32^3).
//
// Same double step as bulk_kernels.cuh in two passes over the spectrum.  A
// line of n = R_1 R_2 ... R_S points is transformed in place in shared
// memory, one stage per radix: stage s takes the R_s points at stride M / R_s
// of each block of M points (M = n, n / R_1, ...), transforms them in
// registers and writes them back where they were, times W_M^(j k).  Frequency
// k = k_1 + R_1 (k_2 + R_2 (...)) ends at position (... (k_1) R_2 + k_2) R_3
// + ...; the inverse runs the stages backwards from there.  Nothing is
// reordered in between: the diffusion factors are tabulated by position, and
// position 0 is frequency 0.
//
// The y transform is cut between two of its stages.  Its first stages couple
// the R_o rows y = j + M' r of a z plane (M' = gy / R_o), its last ones the M'
// neighbouring rows of a block of positions, so
//   k_mx_a (one block per row set (j, z)): outer inverse y stages, inverse x,
//          node t of both chains, forward x, outer forward y stages;
//   k_mx_b (one block per (row block, columns)): inner y stages, forward z,
//          exp(-ds k^2) / N, inverse z, inner inverse y stages
// are a whole double step: the spectrum is read and written twice, by blocks
// of a few hundred to a few thousand points whatever the grid.  Butterflies
// are compile-time radices up to 16 behind a switch that is uniform over the
// block; the outermost stages of a pass read and write global memory.
//
// The FP32 (0, 0) pencil (see DcPencil): k_mx_a leaves every row's kx = 0
// entry in dcin, blocks of their own in k_mx_b add them up over y and convolve
// the sums into dcout, the table's factor of that pencil is zero, and the next
// k_mx_a adds dcout to the kx = 0 entry of every row.  Neither the cut nor the
// launch geometry changes an operation, so the tuner's choice does not either.
//
// Bound: FP32 the latency of the stages (a barrier each), FP64 the FP64 pipe:
// one warp instruction per 64 cycles on each SM quarter, so FP64 plans with
// fewer points than lanes take small radices, which leave every quarter a
// short program.
#pragma once
#include <vector>

#include "bulk_tma.cuh"

struct adscf_ctx;

namespace mxk {

constexpr int kMaxStages = 6;
struct Axis {                   // radices and block lengths of an axis's stages
  int n, nst, tw_off;
  int rad[kMaxStages], m[kMaxStages];
};

// One stage over `lines` lines of a tile.  Task t: line l = t mod lines, then
// b = u / mp, j = u mod mp of u = t / lines; its points are b m + j + r mp.
struct Step {
  int R, m, mp, total;          // radix, block length and stride in the tile, tasks
  unsigned mg, mgl;             // 2^20 / mp + 1, div_magic(lines)
  int lines, lmask, lsh;        // line l at (l & lmask) ls + (l >> lsh) ls2
  int ls, ls2, es;              // pitches in shared memory
  int gls, gls2, ges;           // pitches in global memory (first and last steps)
  int tw, tws, jmul, jin;       // twiddle table, W index = (jmul j + jin tile j) tws k
};
constexpr int kMaxSteps = 8;
// stage before a step's one on its axis: radix (0: none) and twiddle step, and
// the blocks of the step's length in a tile; for the steps of both programs and
// the z visit (bulk_mx_spread.cuh)
struct Prev {
  int rp, twp, nb;
};
struct Spread {
  Prev a[kMaxSteps], b[kMaxSteps];
  int zrp, ztwp;
};
struct Prog {
  int n;
  Step s[kMaxSteps];            // in forward order
};

// Arrays of one context
template <typename T>
struct Io {
  const T* fk;                  // by position: g_xy hi, lo [gy gx] each, g_z / N hi, lo [gz] each
  const BulkDev<T>* I;
  cplx<T>* spec;
  cplx<T>* slices;
  const T* E;
  float2* dcin;                 // [gz][gy] FP32 kx = 0 entries of the rows before the y and z transforms
  float2* dcout;                // [gz] the pencil convolved by the z pass
  const float2* dcc;            // [gz] its kernel, (hi, lo)
};

template <typename T>
struct Dev {
  int gx, gy, gz;
  int ro, mi;                   // outer rows of a tile (R_o), rows of an inner block (M')
  int pitch;                    // row pitch of k_mx_a's tile (odd)
  int cols, lc, ctiles;         // columns of k_mx_b's tile (a power of two, its log), tiles along x
  int pb;                       // pitch of its rows, [y'][z][column]
  int stream;                   // FP32: factors and slices past L2's eviction order
  int ntiles;                   // blocks of columns of k_mx_b (the rest convolve the pencil)
  Prog a, b;                    // steps around the real-space visit / the diffusion factor
  int rx, rz;                   // radices of those visits (1: none)
  int nxs;                      // x steps of program a (its first ones)
  unsigned mgj, mgz;            // divisions by gx / rx, and by the z lines of a tile
  int tw_x, tw_y, tw_z;         // twiddle tables in `tw`
  const cplx<T>* tw;
  Io<T> io;
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

// One stage of the tile: forward (SG = 1) transforms, then multiplies by
// W^(j k); inverse (SG = -1) multiplies by the conjugate, then transforms.
// g: global memory the points come from (inverse of k_mx_a, forward of
// k_mx_b) or go to, null for shared memory; lines with (l & lmask) >= nl do
// not exist there.  dc (the x step next to the row's end, FP32): value added
// to point 0 of every line (SG < 0), or where point 0 of line l is left, at
// dc[l dcs] (SG > 0).
template <typename T, int SG, bool SRC, int R>
__device__ __forceinline__ void stage_r(const Step& S, cplx<T>* sm, int tile_j, cplx<T>* g, int nl, float2* dc,
                                        int dcs) {
  for (int t = threadIdx.x; t < S.total; t += blockDim.x) {
    const int u = fdiv(t, S.mgl), l = t - u * S.lines;
    const int b = (int)(((unsigned)u * S.mg) >> 20), j = u - b * S.mp;
    const int at = b * S.m + j, lo = l & S.lmask, hi = l >> S.lsh;
    cplx<T>* p = sm + lo * S.ls + hi * S.ls2 + at * S.es;
    cplx<T>* q = g ? g + (size_t)lo * S.gls + (size_t)hi * S.gls2 + (size_t)at * S.ges : nullptr;
    const int st = S.mp * S.es;
    const size_t gst = (size_t)S.mp * S.ges;
    cplx<T> v[R];
    if (SRC && g) {
      if (lo < nl) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = q[r * gst];
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = mk<T>((T)0, (T)0);
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * st];
    }
    if constexpr (sizeof(T) == 4 && SG < 0)
      if (dc && at == 0) v[0] = cadd<T>(v[0], *dc);
    const int ji = (S.jmul * j + S.jin * tile_j) * S.tws;
    const cplx<T>* w = sm + S.tw;
    if (SG < 0 && ji) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmulc<T>(v[r], w[ji * r]);
    }
    dft<T, R>(v, SG);
    if (SG > 0 && ji) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul<T>(v[r], w[ji * r]);
    }
    if constexpr (sizeof(T) == 4 && SG > 0)
      if (dc && at == 0) dc[(size_t)l * dcs] = v[0];
    if (!SRC && g) {
      if (lo < nl) {
#pragma unroll
        for (int r = 0; r < R; ++r) q[r * gst] = v[r];
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) p[r * st] = v[r];
    }
  }
}

// What the visit of the diffusion factor does besides, for the adjoint: the
// forward pass keeps its spectra (kStore), the reverse pass adds Re(conj(kept)
// spectrum) up per frequency (kDot), from spectra that were kept or are made again
// from the slices (kSpec: the spectrum alone, nothing after it).  All lie in tile
// order: point (row yy, position zp, column c) of a block at ((zp M' + yy) cols + c).
enum { kPlain = 0, kStore = 1, kDot = 2, kSpec = 3 };
template <typename T>
struct Side {
  cplx<T>* keep;                // the block's part of the kept spectrum
  double* dot;                  // and of the sums
};

// Last forward stage, diffusion factor and first inverse stage of the z lines
// in one visit of the points (both stages have M = R, no twiddles).  Lines
// (row yy of the block, column c); fz: the g_z / N factors by position (hi
// [n], lo [n]); fxy: the tile's g_xy (rows gx apart, lo parts at + nxy).
template <typename T, int R, int MODE = kPlain>
__device__ __forceinline__ void mid_r(const Dev<T>& D, cplx<T>* sm, const T* fz, const T* fxy, int nl,
                                      const Side<T>& sd = Side<T>{}) {
  const int gz = D.gz, lines = D.mi << D.lc, nxy = D.gx * D.gy;
  const int total = gz / R * lines;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int u = fdiv(t, D.mgz), l = t - u * lines;
    const int c = l & (D.cols - 1), yy = l >> D.lc;
    if (c >= nl) continue;
    cplx<T>* p = sm + yy * D.pb + ((u * R) << D.lc) + c;
    const T ah = __ldg(fxy + (size_t)yy * D.gx + c);
    T al = (T)0;
    if constexpr (sizeof(T) == 4) al = __ldg(fxy + nxy + (size_t)yy * D.gx + c);
    cplx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[r << D.lc];
    if constexpr (R > 1) dft<T, R>(v, +1);
    if constexpr (MODE != kPlain) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const size_t at = (size_t)(((u * R + r) * D.mi + yy) << D.lc) + c;
        if constexpr (MODE != kDot) {
          sd.keep[at] = v[r];
        } else {
          const cplx<T> f = sd.keep[at];
          sd.dot[at] += f.x * v[r].x + f.y * v[r].y;
        }
      }
    }
    if constexpr (MODE == kSpec) continue;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const T bh = fz[u * R + r];
      if constexpr (sizeof(T) == 4) {   // compensated product, one rounding
        const float bl = fz[gz + u * R + r];
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
    for (int r = 0; r < R; ++r) p[r << D.lc] = v[r];
  }
}

// Boltzmann factors of a point
template <typename T>
__device__ __forceinline__ EPt<T> load_e(const Dev<T>& D, const T* E, size_t p) {
  if constexpr (sizeof(T) == 4)
    if (D.stream) {
      const float4 v = __ldcs(reinterpret_cast<const float4*>(E) + p);
      return {v.x, v.y, v.z, v.w};
    }
  return load_ept(E, p);
}

// Last inverse stage of the x rows, node t of both chains and the first
// forward stage in one visit (both stages have M = n: a task holds points
// j + r n / R of a row; tasks of a row are neighbours, so the Boltzmann
// factors and the slice move in runs of n / R points).  E, sl: factors and
// slice at the tile's first row, its rows M' gx apart; f: bits 0-3 = forward /
// backward chain takes the A factor at node t, at node t + 1; bit 4: t <
// Ns, the forward stage follows; init: no inverse, slice = (1, 1); dco, dci:
// as dc of stage_r where this is the rows' only stage, else null.  FROM: no
// inverse, node t is the slice.
template <typename T, int R, bool FROM = false>
__device__ __forceinline__ void real_r(const Dev<T>& D, cplx<T>* sm, const T* E, cplx<T>* sl, unsigned f, bool init,
                                       float2* dco, float2* dci) {
  const int Mp = D.gx / R;
  const int total = Mp * D.ro;
  const size_t rs = (size_t)D.mi * D.gx;
  const bool fA = f & 1, bA = f & 2, fA2 = f & 4, bA2 = f & 8, more = f & 16;
  const cplx<T>* w = sm + D.ro * D.pitch;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int l = fdiv(t, D.mgj), j = t - l * Mp;
    cplx<T>* p = sm + l * D.pitch + j;
    const size_t gp = l * rs + j;
    cplx<T> v[R];
    if (!FROM && !init) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * Mp];
      if constexpr (sizeof(T) == 4)
        if (dco) v[0] = cadd<T>(v[0], *dco);   // the only stage: j = 0
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
      const EPt<T> ev = load_e(D, E, gp + r * Mp);
      if constexpr (FROM) {
        const cplx<T> q = sl[gp + r * Mp];
        v[r] = mk<T>(emul(q.x, fA2 ? ev.a : ev.b, fA2 ? ev.al : ev.bl),
                     emul(q.y, bA2 ? ev.a : ev.b, bA2 ? ev.al : ev.bl));
      } else if (init) {
        v[r] = mk<T>(fA ? ev.a : ev.b, bA ? ev.a : ev.b);
        sl[gp + r * Mp] = mk<T>((T)1, (T)1);
      } else {
        const cplx<T> q = mk<T>(emul(v[r].x, fA ? ev.a : ev.b, fA ? ev.al : ev.bl),
                                emul(v[r].y, bA ? ev.a : ev.b, bA ? ev.al : ev.bl));
        if (sizeof(T) == 4 && D.stream) __stcs(sl + gp + r * Mp, q);
        else sl[gp + r * Mp] = q;
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
    if constexpr (sizeof(T) == 4)
      if (dci) dci[(size_t)l * D.mi] = v[0];
#pragma unroll
    for (int r = 0; r < R; ++r) p[r * Mp] = v[r];
  }
}

}  // namespace mxk

// ---------------------------------------------------------------------------
// Real-space pass of the row set (j, z): block j + M' z.  t = 0 starts the
// chains: slice 0 = (1, 1).  FROM: the pass after node t, from its slice.  Shared
// memory: R_o pitch + gx + gy points.
// ---------------------------------------------------------------------------
template <typename T, bool FROM = false>
__device__ __forceinline__ void mx_a_body(const mxk::Dev<T>& D, const mxk::Io<T>& io, int t) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
  const BulkDev<T>& I = *io.I;
  const int gx = D.gx, ro = D.ro, mi = D.mi;
  const int z = blockIdx.x / mi, j = blockIdx.x - z * mi;
  const size_t base = ((size_t)z * D.gy + j) * gx;
  const size_t rs = (size_t)mi * gx;
  const int ns = I.ns;
  tmak::pdl_launch_dependents();
  {
    cplx<T>* tw = sm + ro * D.pitch;
    for (int i = threadIdx.x; i < gx; i += blockDim.x) tw[i] = D.tw[D.tw_x + i];
    if (ro > 1)
      for (int i = threadIdx.x; i < D.gy; i += blockDim.x) tw[gx + i] = D.tw[D.tw_y + i];
  }
  const int tt = t == 0 ? 1 : t;
  const bool more = t == 0 || t < ns;
  const unsigned f = (chain_type_fwd(I, tt) == 0 ? 1u : 0u) | (chain_type_bwd(I, tt) == 0 ? 2u : 0u) |
                     (chain_type_fwd(I, t + 1) == 0 ? 4u : 0u) | (chain_type_bwd(I, t + 1) == 0 ? 8u : 0u) |
                     (more ? 16u : 0u);
  cplx<T>* sl = io.slices + (size_t)t * (size_t)I.npts + base;
  const T* E = io.E + base * (sizeof(T) == 4 ? 4 : 2);
  cplx<T>* g = io.spec + base;
  // the x step where a row's kx = 0 entry is complete (none: the real visit)
  const int xs = sizeof(T) == 4 ? D.nxs - 1 : -2;
  float2* dci = sizeof(T) == 4 ? io.dcin + (size_t)z * D.gy + j : nullptr;
  float2* dco = sizeof(T) == 4 ? io.dcout + z : nullptr;
  tmak::pdl_wait();
  __syncthreads();
  if (!FROM && t > 0) {
    // the tile's Boltzmann factors on their way to L1 while it is transformed
    for (int r = 0; r < ro; ++r) {
      const char* e0 = reinterpret_cast<const char*>(E) + r * rs * 16;
      for (int i = threadIdx.x * 128; i < gx * 16; i += blockDim.x * 128) tmak::prefetch_l1(e0 + i);
    }
    if (D.a.n == 0) {
      for (int x = threadIdx.x; x < gx; x += blockDim.x) sm[x] = g[x];
      __syncthreads();
    }
    for (int i = D.a.n - 1; i >= 0; --i) {
      const mxk::Step& S = D.a.s[i];
      cplx<T>* src = i == D.a.n - 1 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::stage_r<T, -1, true, R_>(S, sm, j, src, gx, i == xs ? dco : nullptr, 0)
      ADSCF_MX_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
      __syncthreads();
    }
  }
  if (D.rx == 1) {
    mxk::real_r<T, 1, FROM>(D, sm, E, sl, f, t == 0, xs == -1 ? dco : nullptr, xs == -1 ? dci : nullptr);
  } else {
#define ADSCF_MX_CALL(R_) \
  mxk::real_r<T, R_, FROM>(D, sm, E, sl, f, t == 0, xs == -1 ? dco : nullptr, xs == -1 ? dci : nullptr)
    ADSCF_MX_SWITCH(D.rx, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
  }
  if (!more) return;
  __syncthreads();
  for (int i = 0; i < D.a.n; ++i) {
    const mxk::Step& S = D.a.s[i];
    cplx<T>* dst = i == D.a.n - 1 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::stage_r<T, +1, false, R_>(S, sm, j, dst, gx, i == xs ? dci : nullptr, mi)
    ADSCF_MX_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
    if (!dst) __syncthreads();
  }
  if (D.a.n == 0) {
    __syncthreads();
    for (int x = threadIdx.x; x < gx; x += blockDim.x) g[x] = sm[x];
  }
}

template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 6 : 4)
k_mx_a(const __grid_constant__ mxk::Dev<T> D, int t) {
  mx_a_body<T>(D, D.io, t);
}
// Contexts blockIdx.y of a batch that share D's grid.  Their arrays come from a
// struct in memory where k_mx_a has kernel parameters, and at the same registers
// (blocks an SM) the pointers spill: 140 bytes here, 392 in k_mx_b_b<float, 256>, of
// k_mx_a's 0 and k_mx_b's 20.
template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 6 : 4)
k_mx_a_b(const __grid_constant__ mxk::Dev<T> D, const mxk::Io<T>* __restrict__ ios, int t) {
  mx_a_body<T>(D, ios[blockIdx.y], t);
}

// ---------------------------------------------------------------------------
// Diffusion pass of the row block k (positions [k M', (k + 1) M') of y) and a
// tile of `cols` columns: block k ctiles + tile.  Blocks from ntiles on: one
// output of the FP32 (0, 0) pencil per warp.  Shared memory: M' gz cols + gy
// + gz points and 2 gz factors.
// ---------------------------------------------------------------------------
template <typename T, int MODE>
__device__ __forceinline__ void mx_b_body(const mxk::Dev<T>& D, const mxk::Io<T>& io, const mxk::Side<T>& sd) {
  extern __shared__ __align__(16) unsigned char smraw[];
  cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
  const int gx = D.gx, gz = D.gz, mi = D.mi, nxy = gx * D.gy;
  tmak::pdl_launch_dependents();
  if constexpr (sizeof(T) == 4) {
    if ((int)blockIdx.x >= D.ntiles) {
      float2* in = reinterpret_cast<float2*>(smraw);
      float2* c = in + ((gz + 1) & ~1);
      for (int i = threadIdx.x; i < gz; i += blockDim.x) c[i] = io.dcc[i];
      tmak::pdl_wait();
      // row sums in float-float, eight threads per plane (rows y = k, k + 8,
      // ... each, then over k): many loads are in flight
      constexpr int kParts = 8;
      float4* part = reinterpret_cast<float4*>(c + ((gz + 1) & ~1));
      for (int i = threadIdx.x; i < gz * kParts; i += blockDim.x) {
        float xh = 0.f, xl = 0.f, yh = 0.f, yl = 0.f;
        const float2* row = io.dcin + (size_t)(i / kParts) * D.gy;
#pragma unroll 4
        for (int y = i % kParts; y < D.gy; y += kParts) {
          const float2 v = row[y];
          ff_add(xh, xl, v.x, 0.f);
          ff_add(yh, yl, v.y, 0.f);
        }
        part[i] = make_float4(xh, xl, yh, yl);
      }
      __syncthreads();
      for (int i = threadIdx.x; i < gz; i += blockDim.x) {
        float4 s = part[i * kParts];
#pragma unroll
        for (int k = 1; k < kParts; ++k) {
          const float4 v = part[i * kParts + k];
          ff_add(s.x, s.y, v.x, v.y);
          ff_add(s.z, s.w, v.z, v.w);
        }
        in[i] = make_float2(s.x + s.y, s.z + s.w);
      }
      __syncthreads();
      const int z = ((int)blockIdx.x - D.ntiles) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      if (z < gz) {
        const float2 o = tmak::dc_point(in, c, gz, z);
        if ((threadIdx.x & 31) == 0) io.dcout[z] = o;
      }
      return;
    }
  }
  const int k = blockIdx.x / D.ctiles, c0 = (blockIdx.x - k * D.ctiles) << D.lc;
  const int nl = min(D.cols, gx - c0);
  const int pts = mi * D.pb;
  T* fz = reinterpret_cast<T*>(sm + pts + D.gy + gz);
  if (mi > 1)
    for (int i = threadIdx.x; i < D.gy; i += blockDim.x) sm[pts + i] = D.tw[D.tw_y + i];
  for (int i = threadIdx.x; i < gz; i += blockDim.x) sm[pts + D.gy + i] = D.tw[D.tw_z + i];
  {
    const T* gzt = io.fk + 2 * (size_t)nxy;
    for (int i = threadIdx.x; i < 2 * gz; i += blockDim.x) fz[i] = gzt[i];
  }
  cplx<T>* g = io.spec + (size_t)k * mi * gx + c0;
  const T* fxy = io.fk + (size_t)k * mi * gx + c0;
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
    cplx<T>* src = i == 0 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::stage_r<T, +1, true, R_>(S, sm, 0, src, nl, nullptr, 0)
    ADSCF_MX_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
    __syncthreads();
  }
  if (D.rz == 1) {
    mxk::mid_r<T, 1, MODE>(D, sm, fz, fxy, nl, sd);
  } else {
#define ADSCF_MX_CALL(R_) mxk::mid_r<T, R_, MODE>(D, sm, fz, fxy, nl, sd)
    ADSCF_MX_SWITCH(D.rz, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
  }
  if constexpr (MODE == mxk::kSpec) return;
  __syncthreads();
  for (int i = D.b.n - 1; i >= 0; --i) {
    const mxk::Step& S = D.b.s[i];
    cplx<T>* dst = i == 0 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::stage_r<T, -1, false, R_>(S, sm, 0, dst, nl, nullptr, 0)
    ADSCF_MX_SWITCH(S.R, ADSCF_MX_CALL)
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
template <typename T, int BT>
__global__ void __launch_bounds__(BT, BT == 512 ? 1 : sizeof(T) == 4 ? 3 : 2)
k_mx_b(const __grid_constant__ mxk::Dev<T> D) {
  mx_b_body<T, mxk::kPlain>(D, D.io, mxk::Side<T>{});
}
template <typename T, int BT>
__global__ void __launch_bounds__(BT, BT == 512 ? 1 : sizeof(T) == 4 ? 3 : 2)
k_mx_b_b(const __grid_constant__ mxk::Dev<T> D, const mxk::Io<T>* __restrict__ ios) {
  mx_b_body<T, mxk::kPlain>(D, ios[blockIdx.y], mxk::Side<T>{});
}

// Plan of a context for launches from another file
struct MxLaunch64 {
  mxk::Dev<double> D;
  bool yz;                      // D's y axis is the grid's z axis
  int thr_a, thr_b, grid_a, grid_b;
  size_t sm_a, sm_b;
  int optin;
  bool spread;                  // its chains run the kernels with an output per lane
  mxk::Spread sp;
  int thr_as, thr_bs;
};
bool mx_launch64(const adscf_ctx* ctx, MxLaunch64& L);   // false: the context has no such plan
// those kernels with side data (mode kStore or kSpec), and the real-space pass after
// node t from its slice
void mx_spread_b_side(const MxLaunch64& L, int mode, double2* keep, int tile, cudaStream_t s);
void mx_spread_a_from(const MxLaunch64& L, int t, cudaStream_t s);
void mx_freqs(const adscf_ctx* ctx, std::vector<int>& f);   // frequency by position, x then y then z

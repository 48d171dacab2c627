// adjoint_mx.cuh -- the reverse sweep of adjoint_kernels.cuh on the mixed-radix
// passes (bulk_mx.cuh).
//
// The gradient needs the spectrum of every step after its forward transform,
// Xf(t) = FFT(E(t) z_{t-1}), in the order in which the diffusion pass holds it.
// Forward passes for a gradient keep them where they take little of the memory
// (adj_mx_keep), and the reverse sweep transforms the adjoint pair alone, six line
// transforms a step for nine.  A sweep behind a forward pass that kept none makes
// them again from the slices, with the forward
// pass's own operations (k_mx_a_from, or its counterpart with an output per lane, and
// kSpec), so that the gradient is the same bits.  Two passes like a forward step:
//   k_mx_adj_a(t): inverse y and x of the adjoint spectrum -> E(t+1) -> + seeds
//                  -> E(t) -> forward x and y;
//   k_mx_b, kDot : forward y and z, W(k) += Re(conj(Xf(t, k)) Ya(t, k)), G / M,
//                  inverse z and y.
// The box gradient is linear in W: g_c = sum_k k_c^2 G(k) / M W(k), once at the
// end (k_mx_adj_sum), so a step spends two FP64 operations a point on it.
//
// Bound: the FP64 pipe.  64^3, 96 steps, forward and backward: 15.8 ms, against
// 26.6 ms with nine transforms on the generic passes.
#pragma once
#include "adjoint_kernels.cuh"
#include "bulk_mx.cuh"

namespace mxk {

// Real-space visit of the reverse sweep (as real_r): E, b, sl: factors,
// cotangents and mirror node at the tile's first row; f: bits 0-3 as real_r's
// for nodes t (0, 1) and t + 1 (2, 3); c: contour weights of nodes t and Ns - t;
// first: t = Ns, no adjoint state yet.
struct Seeds {
  double cat, cbt, cau, cbu, aS;
};
template <int R>
__device__ __forceinline__ void adj_real_r(const Dev<double>& D, double2* sm, const double* E, const double* b,
                                           const double2* sl, size_t np, unsigned f, bool first, const Seeds& c) {
  const int Mp = D.gx / R;
  const int total = Mp * D.ro;
  const size_t rs = (size_t)D.mi * D.gx;
  const bool fA = f & 1, bA = f & 2, fA1 = f & 4, bA1 = f & 8;
  const double2* w = sm + D.ro * D.pitch;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int l = fdiv(t, D.mgj), j = t - l * Mp;
    double2* p = sm + l * D.pitch + j;
    const size_t gp = l * rs + j;
    double2 v[R];
    if (!first) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * Mp];
      if constexpr (R > 1) {
        if (j) {
#pragma unroll
          for (int r = 1; r < R; ++r) v[r] = cmulc<double>(v[r], w[j * r]);
        }
        dft<double, R>(v, -1);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const size_t g = gp + r * Mp;
      const EPt<double> ev = load_ept(E, g);
      const double2 s2 = __ldg(sl + g);   // (q_{Ns-t}, qdag_{Ns-t})
      const double ba = __ldg(b + g), bb = __ldg(b + np + g);
      double lam = c.aS, mu = 0.0;
      if (!first) {
        lam = v[r].x * (fA1 ? ev.a : ev.b);
        mu = v[r].y * (bA1 ? ev.a : ev.b);
      }
      lam += (c.cat * ba + c.cbt * bb) * s2.y;
      mu += (c.cau * ba + c.cbu * bb) * s2.x;
      v[r] = make_double2(lam * (fA ? ev.a : ev.b), mu * (bA ? ev.a : ev.b));
    }
    if constexpr (R > 1) {
      dft<double, R>(v, +1);
      if (j) {
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul<double>(v[r], w[j * r]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) p[r * Mp] = v[r];
  }
}

}  // namespace mxk

// Real-space pass of step t of the reverse sweep on the row set (j, z), as
// k_mx_a
static __global__ void __launch_bounds__(128, 4)
k_mx_adj_a(const __grid_constant__ mxk::Dev<double> D, const double* __restrict__ b, const double* __restrict__ sc,
           int t) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sm = reinterpret_cast<double2*>(smraw);
  const BulkDev<double>& I = *D.io.I;
  const int gx = D.gx, ro = D.ro, mi = D.mi;
  const int z = blockIdx.x / mi, j = blockIdx.x - z * mi;
  const size_t base = ((size_t)z * D.gy + j) * gx, rs = (size_t)mi * gx;
  {
    double2* tw = sm + ro * D.pitch;
    for (int i = threadIdx.x; i < gx; i += blockDim.x) tw[i] = D.tw[D.tw_x + i];
    if (ro > 1)
      for (int i = threadIdx.x; i < D.gy; i += blockDim.x) tw[gx + i] = D.tw[D.tw_y + i];
  }
  const bool first = t == I.ns;
  const int u = I.ns - t;
  const unsigned f = (chain_type_fwd(I, t) == 0 ? 1u : 0u) | (chain_type_bwd(I, t) == 0 ? 2u : 0u) |
                     (chain_type_fwd(I, t + 1) == 0 ? 4u : 0u) | (chain_type_bwd(I, t + 1) == 0 ? 8u : 0u);
  const float2 wt = node_weights(I, t), wu = node_weights(I, u);
  const mxk::Seeds c{I.ds * (double)wt.x, I.ds * (double)wt.y, I.ds * (double)wu.x, I.ds * (double)wu.y,
                     first ? sc[ADJ_AS] : 0.0};
  const double2* sl = D.io.slices + (size_t)u * (size_t)I.npts + base;
  const double* E = D.io.E + base * 2;
  double2* g = D.io.spec + base;
  __syncthreads();
  if (!first) {
    for (int r = 0; r < ro; ++r) {   // the tile's factors on their way to L1
      const char* e0 = reinterpret_cast<const char*>(E) + r * rs * 16;
      for (int i = threadIdx.x * 128; i < gx * 16; i += blockDim.x * 128) tmak::prefetch_l1(e0 + i);
    }
    if (D.a.n == 0) {
      for (int x = threadIdx.x; x < gx; x += blockDim.x) sm[x] = g[x];
      __syncthreads();
    }
    for (int i = D.a.n - 1; i >= 0; --i) {
      const mxk::Step& S = D.a.s[i];
      double2* src = i == D.a.n - 1 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::stage_r<double, -1, true, R_>(S, sm, j, src, gx, nullptr, 0)
      ADSCF_MX_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
      __syncthreads();
    }
  }
  if (D.rx == 1) {
    mxk::adj_real_r<1>(D, sm, E, b + base, sl, (size_t)I.npts, f, first, c);
  } else {
#define ADSCF_MX_CALL(R_) mxk::adj_real_r<R_>(D, sm, E, b + base, sl, (size_t)I.npts, f, first, c)
    ADSCF_MX_SWITCH(D.rx, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
  }
  __syncthreads();
  for (int i = 0; i < D.a.n; ++i) {
    const mxk::Step& S = D.a.s[i];
    double2* dst = i == D.a.n - 1 ? g : nullptr;
#define ADSCF_MX_CALL(R_) mxk::stage_r<double, +1, false, R_>(S, sm, j, dst, gx, nullptr, 0)
    ADSCF_MX_SWITCH(S.R, ADSCF_MX_CALL)
#undef ADSCF_MX_CALL
    if (!dst) __syncthreads();
  }
  if (D.a.n == 0)
    for (int x = threadIdx.x; x < gx; x += blockDim.x) g[x] = sm[x];
}

// Real-space pass after node t of the chains, from its slice, into D.io.spec
static __global__ void __launch_bounds__(128, 4) k_mx_a_from(const __grid_constant__ mxk::Dev<double> D, int t) {
  mx_a_body<double, true>(D, D.io, t);
}

// Diffusion pass with side data of `tile` points a block
template <int BT, int MODE>
__global__ void __launch_bounds__(BT, BT == 512 ? 1 : 2)
k_mx_b_side(const __grid_constant__ mxk::Dev<double> D, double2* keep, double* dot, int tile) {
  const size_t at = (size_t)blockIdx.x * tile;
  mx_b_body<double, MODE>(D, D.io, mxk::Side<double>{keep + at, dot ? dot + at : nullptr});
}

// Block sums of k_c^2 G(k) / M W(k) for c = x, y, z into gpart[block][3];
// frq: frequency by position (x, then y, then z); yz: D's y axis is the grid's z
// axis, lx, ly, lz are D's
static __global__ void __launch_bounds__(256)
k_mx_adj_sum(const __grid_constant__ mxk::Dev<double> D, const double* __restrict__ dot, const int* __restrict__ frq,
             int tile, bool yz, double lx, double ly, double lz, double* __restrict__ gpart) {
  __shared__ double red[3 * 32];
  const int gx = D.gx, gy = D.gy, mi = D.mi;
  const int k = blockIdx.x / D.ctiles, c0 = (blockIdx.x - k * D.ctiles) << D.lc;
  const double* w = dot + (size_t)blockIdx.x * tile;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int e = threadIdx.x; e < tile; e += blockDim.x) {
    const int x = c0 + (e & (D.cols - 1)), r = e >> D.lc, zp = r / mi, y = k * mi + r - zp * mi;
    if (x >= gx) continue;
    const double v = w[e] * (D.io.fk[(size_t)y * gx + x] * D.io.fk[2 * (size_t)gx * gy + zp]);
    acc[0] += v * adj_k2(frq[x], gx, lx);
    acc[1] += v * adj_k2(frq[gx + y], gy, ly);
    acc[2] += v * adj_k2(frq[gx + gy + zp], D.gz, lz);
  }
  const double s = block_reduce_k<3>(acc, red);
  if (threadIdx.x < 3) gpart[blockIdx.x * 3 + (yz && threadIdx.x ? 3 - threadIdx.x : threadIdx.x)] = s;
}

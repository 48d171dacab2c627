// adjoint_mx.cu -- forward pass with kept spectra and reverse sweep on the
// mixed-radix passes (adjoint_mx.cuh).
#include <algorithm>
#include <vector>

#include "internal.h"
#include "adjoint_mx.cuh"
#include "adjoint_mx_host.h"

namespace {

template <int MODE>
void step_b(const MxLaunch64& L, double2* keep, double* dot, int tile, cudaStream_t s) {
  if constexpr (MODE != mxk::kDot) {
    if (L.spread) {
      mx_spread_b_side(L, MODE, keep, tile, s);
      return;
    }
  }
  if (L.thr_b > 256) k_mx_b_side<512, MODE><<<L.grid_b, L.thr_b, L.sm_b, s>>>(L.D, keep, dot, tile);
  else k_mx_b_side<256, MODE><<<L.grid_b, L.thr_b, L.sm_b, s>>>(L.D, keep, dot, tile);
}

// the spectrum of step t from slice t - 1
void spectrum(MxLaunch64 L, double2* spec2, double2* one, int tile, int t, cudaStream_t s) {
  L.D.io.spec = spec2;
  if (L.spread) mx_spread_a_from(L, t - 1, s);
  else k_mx_a_from<<<L.grid_a, L.thr_a, L.sm_a, s>>>(L.D, t - 1);
  step_b<mxk::kSpec>(L, one, nullptr, tile, s);
}

// Spectra of all steps, as much memory as the slices: up to 1 GB from the first
// forward pass on (64^3, 100 steps 0.4 GB; forward and reverse 15.9 ms, 20.5 with the
// spectra made again), larger ones, which a program that only evaluates free energies
// should not pay for, from the first reverse sweep on (`sweep`), where they take at
// most a quarter of the free memory and a sixteenth of the GPU's.  Tried once.
int adj_mx_keep(adscf_ctx* ctx, AdjMx* X, const MxLaunch64& L, bool sweep) {
  X->tile = (L.D.mi * L.D.gz) << L.D.lc;
  X->ntiles = L.D.ntiles;
  X->pts = (size_t)X->tile * X->ntiles;
  const size_t bytes = X->pts * ctx->ns * sizeof(double2);
  if (X->tried || (!sweep && bytes > (size_t(1) << 30))) return ADSCF_OK;
  X->tried = true;
  size_t avail = 0, total = 0;
  CK(cudaMemGetInfo(&avail, &total));
  if (bytes <= std::min(avail / 4, total / 16) && cudaMalloc(&X->keep, bytes)) {
    cudaGetLastError();
    X->keep = nullptr;
  }
  auto set = [&](auto* k) { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, L.optin); };
  CK(set(k_mx_b_side<256, mxk::kStore>));
  CK(set(k_mx_b_side<512, mxk::kStore>));
  return ADSCF_OK;
}

// buffers of the reverse sweep
int adj_mx_setup(adscf_ctx* ctx, AdjMx* X, const MxLaunch64& L) {
  const int rc = adj_mx_keep(ctx, X, L, true);
  if (rc || X->dot) return rc;
  const size_t pts = X->pts;
  std::vector<int> f;
  mx_freqs(ctx, f);
  if (cudaMalloc(&X->one, pts * sizeof(double2)) || cudaMalloc(&X->dot, pts * sizeof(double)) ||
      cudaMalloc(&X->gpart, 3 * (size_t)L.D.ntiles * sizeof(double)) || cudaMalloc(&X->frq, f.size() * sizeof(int))) {
    cudaGetLastError();
    cudaFree(X->one); cudaFree(X->dot); cudaFree(X->gpart);
    X->one = nullptr; X->dot = X->gpart = nullptr;
    return set_err(ctx, ADSCF_E_OOM, "adjoint buffers");
  }
  CK(cudaMemcpy(X->frq, f.data(), f.size() * sizeof(int), cudaMemcpyHostToDevice));
  auto set = [&](auto* k) { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, L.optin); };
  CK(set(k_mx_adj_a));
  CK(set(k_mx_a_from));
  CK(set(k_mx_b_side<256, mxk::kSpec>));
  CK(set(k_mx_b_side<512, mxk::kSpec>));
  CK(set(k_mx_b_side<256, mxk::kDot>));
  CK(set(k_mx_b_side<512, mxk::kDot>));
  return ADSCF_OK;
}

}  // namespace

void adj_mx_free(AdjMx* X) {
  cudaFree(X->keep); cudaFree(X->one); cudaFree(X->dot); cudaFree(X->gpart); cudaFree(X->frq);
  *X = AdjMx{};
}

int adj_mx_forward(adscf_ctx* ctx, AdjMx* X) {
  MxLaunch64 L;
  if (!mx_launch64(ctx, L)) return set_err(ctx, ADSCF_E_STATE, "adjoint passes");
  const int rc = adj_mx_keep(ctx, X, L, false);
  if (rc) return rc;
  X->kept = X->keep != nullptr;
  if (!X->kept) return bulk_enqueue_propagate(ctx);
  mx_real(ctx, 0);
  for (int t = 1; t <= ctx->ns; ++t) {
    step_b<mxk::kStore>(L, X->keep + (size_t)(t - 1) * X->pts, nullptr, X->tile, ctx->stream);
    mx_real(ctx, t);
  }
  CK(cudaGetLastError());
  return bulk_enqueue_contour(ctx);
}

int adj_mx_backward(adscf_ctx* ctx, AdjMx* X, const double* b, const double* sc, double2* spec2) {
  MxLaunch64 L;
  if (!mx_launch64(ctx, L)) return set_err(ctx, ADSCF_E_STATE, "adjoint passes");
  const int rc = adj_mx_setup(ctx, X, L);
  if (rc) return rc;
  cudaStream_t s = ctx->stream;
  CK(cudaMemsetAsync(X->dot, 0, X->pts * sizeof(double), s));
  for (int t = ctx->ns; t >= 1; --t) {
    double2* xf = X->kept ? X->keep + (size_t)(t - 1) * X->pts : X->one;
    if (!X->kept) spectrum(L, spec2, xf, X->tile, t, s);
    k_mx_adj_a<<<L.grid_a, L.thr_a, L.sm_a, s>>>(L.D, b, sc, t);
    step_b<mxk::kDot>(L, xf, X->dot, X->tile, s);
  }
  k_mx_adj_sum<<<X->ntiles, 256, 0, s>>>(L.D, X->dot, X->frq, X->tile, L.yz, ctx->p.sizex,
                                         L.yz ? ctx->p.sizez : ctx->p.sizey, L.yz ? ctx->p.sizey : ctx->p.sizez,
                                         X->gpart);
  CK(cudaGetLastError());
  return ADSCF_OK;
}

// adjoint_mx.cu -- forward pass with kept spectra and reverse sweep on the
// mixed-radix passes (adjoint_mx.cuh).
#include <vector>

#include "internal.h"
#include "adjoint_mx.cuh"
#include "adjoint_mx_host.h"

namespace {

template <int MODE>
void step_b(const MxLaunch64& L, double2* keep, double* dot, int tile, cudaStream_t s) {
  if (L.thr_b > 256) k_mx_b_side<512, MODE><<<L.grid_b, L.thr_b, L.sm_b, s>>>(L.D, keep, dot, tile);
  else k_mx_b_side<256, MODE><<<L.grid_b, L.thr_b, L.sm_b, s>>>(L.D, keep, dot, tile);
}

}  // namespace

// Spectra of all steps, where they take at most a quarter of the free memory.
// A context that cannot have them recomputes them in the reverse sweep on the
// generic passes (adjoint.cu).
int adj_mx_setup(adscf_ctx* ctx, AdjMx* X) {
  MxLaunch64 L;
  if (ctx->mx_off || !mx_launch64(ctx, L)) {   // a pinned plan runs the generic sweep
    adj_mx_free(X);
    return ADSCF_OK;
  }
  if (X->keep) return ADSCF_OK;
  const int tile = (L.D.mi * L.D.gz) << L.D.lc;
  const size_t pts = (size_t)tile * L.D.ntiles;
  size_t avail = 0, total = 0;
  CK(cudaMemGetInfo(&avail, &total));
  if (pts * ctx->ns * sizeof(double2) > avail / 4) return ADSCF_OK;
  std::vector<int> f;
  mx_freqs(ctx, f);
  if (cudaMalloc(&X->keep, pts * ctx->ns * sizeof(double2)) || cudaMalloc(&X->dot, pts * sizeof(double)) ||
      cudaMalloc(&X->gpart, 3 * (size_t)L.D.ntiles * sizeof(double)) || cudaMalloc(&X->frq, f.size() * sizeof(int))) {
    cudaGetLastError();
    adj_mx_free(X);
    return ADSCF_OK;
  }
  X->tile = tile;
  X->pts = pts;
  X->ntiles = L.D.ntiles;
  CK(cudaMemcpy(X->frq, f.data(), f.size() * sizeof(int), cudaMemcpyHostToDevice));
  CK(cudaFuncSetAttribute(k_mx_adj_a, cudaFuncAttributeMaxDynamicSharedMemorySize, L.optin));
  CK(cudaFuncSetAttribute(k_mx_b_side<256, mxk::kStore>, cudaFuncAttributeMaxDynamicSharedMemorySize, L.optin));
  CK(cudaFuncSetAttribute(k_mx_b_side<512, mxk::kStore>, cudaFuncAttributeMaxDynamicSharedMemorySize, L.optin));
  CK(cudaFuncSetAttribute(k_mx_b_side<256, mxk::kDot>, cudaFuncAttributeMaxDynamicSharedMemorySize, L.optin));
  CK(cudaFuncSetAttribute(k_mx_b_side<512, mxk::kDot>, cudaFuncAttributeMaxDynamicSharedMemorySize, L.optin));
  return ADSCF_OK;
}

void adj_mx_free(AdjMx* X) {
  cudaFree(X->keep); cudaFree(X->dot); cudaFree(X->gpart); cudaFree(X->frq);
  *X = AdjMx{};
}

int adj_mx_forward(adscf_ctx* ctx, AdjMx* X) {
  MxLaunch64 L;
  if (!mx_launch64(ctx, L)) return set_err(ctx, ADSCF_E_STATE, "adjoint passes");
  mx_real_plain(ctx, 0);
  for (int t = 1; t <= ctx->ns; ++t) {
    step_b<mxk::kStore>(L, X->keep + (size_t)(t - 1) * X->pts, nullptr, X->tile, ctx->stream);
    mx_real_plain(ctx, t);
  }
  CK(cudaGetLastError());
  return bulk_enqueue_contour(ctx);
}

// b: [2][npts] cotangents, sc: scalars of the forward pass (device)
int adj_mx_backward(adscf_ctx* ctx, AdjMx* X, const double* b, const double* sc) {
  MxLaunch64 L;
  if (!mx_launch64(ctx, L)) return set_err(ctx, ADSCF_E_STATE, "adjoint passes");
  cudaStream_t s = ctx->stream;
  CK(cudaMemsetAsync(X->dot, 0, X->pts * sizeof(double), s));
  for (int t = ctx->ns; t >= 1; --t) {
    k_mx_adj_a<<<L.grid_a, L.thr_a, L.sm_a, s>>>(L.D, b, sc, t);
    step_b<mxk::kDot>(L, X->keep + (size_t)(t - 1) * X->pts, X->dot, X->tile, s);
  }
  k_mx_adj_sum<<<X->ntiles, 256, 0, s>>>(L.D, X->dot, X->frq, X->tile, L.yz, ctx->p.sizex,
                                         L.yz ? ctx->p.sizez : ctx->p.sizey, L.yz ? ctx->p.sizey : ctx->p.sizez,
                                         X->gpart);
  CK(cudaGetLastError());
  return ADSCF_OK;
}

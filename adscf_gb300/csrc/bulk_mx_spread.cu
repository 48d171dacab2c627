// bulk_mx_spread.cu -- launches of the passes with an output per lane
// (bulk_mx_spread.cuh).
#include "bulk_mx_spread.cuh"
#include "launch_pdl.h"

// Programmatic launches up to 4096 points, whose blocks leave SMs free for the
// next kernel's (16^3 13.1 -> 11.6 us a double step, 32 x 1 x 64 13.5 -> 12.1);
// past that the blocks that wait take FP64 pipes from those that work (20 x 18 x
// 30 18.2 -> 30.1).
static bool early(const mxk::Dev<double>& D) { return D.gx * D.gy * D.gz <= 4096; }

cudaError_t mx_spread_setup(int optin) {
  auto set = [&](auto* k) { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin); };
  cudaError_t e = set(k_mx_a_spread);
  if (!e) e = set(k_mx_a_spread_from);
  if (!e) e = set(k_mx_b_spread);
  if (!e) e = set(k_mx_b_spread_side<mxk::kStore>);
  return e ? e : set(k_mx_b_spread_side<mxk::kSpec>);
}
void mx_spread_a(const mxk::Dev<double>& D, const mxk::Spread& W, int grid, int threads, size_t smem, cudaStream_t s,
                 int t) {
  if (early(D)) launch_pdl(k_mx_a_spread, grid, threads, smem, s, D, W, t);
  else k_mx_a_spread<<<grid, threads, smem, s>>>(D, W, t);
}
void mx_spread_b(const mxk::Dev<double>& D, const mxk::Spread& W, int grid, int threads, size_t smem, cudaStream_t s) {
  if (early(D)) launch_pdl(k_mx_b_spread, grid, threads, smem, s, D, W);
  else k_mx_b_spread<<<grid, threads, smem, s>>>(D, W);
}
void mx_spread_b_side(const MxLaunch64& L, int mode, double2* keep, int tile, cudaStream_t s) {
  const auto kern = mode == mxk::kStore ? k_mx_b_spread_side<mxk::kStore> : k_mx_b_spread_side<mxk::kSpec>;
  kern<<<L.grid_b, L.thr_bs, L.sm_b, s>>>(L.D, L.sp, keep, tile);
}
void mx_spread_a_from(const MxLaunch64& L, int t, cudaStream_t s) {
  k_mx_a_spread_from<<<L.grid_a, L.thr_as, L.sm_a, s>>>(L.D, L.sp, t);
}

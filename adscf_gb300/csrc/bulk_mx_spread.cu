// bulk_mx_spread.cu -- launches of the passes with an output per lane
// (bulk_mx_spread.cuh).
#include "bulk_mx_spread.cuh"

cudaError_t mx_spread_setup(int optin) {
  const cudaError_t e = cudaFuncSetAttribute(k_mx_a_spread, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  return e ? e : cudaFuncSetAttribute(k_mx_b_spread, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
}
void mx_spread_a(const mxk::Dev<double>& D, const mxk::Spread& W, int grid, int threads, size_t smem, cudaStream_t s,
                 int t) {
  k_mx_a_spread<<<grid, threads, smem, s>>>(D, W, t);
}
void mx_spread_b(const mxk::Dev<double>& D, const mxk::Spread& W, int grid, int threads, size_t smem, cudaStream_t s) {
  k_mx_b_spread<<<grid, threads, smem, s>>>(D, W);
}

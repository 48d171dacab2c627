// adjoint_mx_host.h -- buffers and entry points of adjoint_mx.cu.
#pragma once
#include <cstddef>

#include <cuda_runtime.h>

struct AdjMx {
  double2* keep = nullptr;      // [ns][pts] spectra of the steps, in tile order; null: not kept
  double* dot = nullptr;        // [pts]
  double* gpart = nullptr;      // [ntiles][3]
  int* frq = nullptr;           // [gx + gy + gz] frequency by position
  int tile = 0, ntiles = 0;
  size_t pts = 0;
  bool kept = false;            // by the last forward pass
};

struct adscf_ctx;
int adj_mx_setup(adscf_ctx* ctx, AdjMx* X);
void adj_mx_free(AdjMx* X);
int adj_mx_forward(adscf_ctx* ctx, AdjMx* X);   // chains, spectra and contour integral
int adj_mx_backward(adscf_ctx* ctx, AdjMx* X, const double* b, const double* sc);

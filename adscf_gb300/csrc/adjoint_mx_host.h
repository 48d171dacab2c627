// adjoint_mx_host.h -- buffers and entry points of adjoint_mx.cu.
#pragma once
#include <cstddef>

#include <cuda_runtime.h>

struct AdjMx {
  bool on = false;              // the last forward pass ran the mixed-radix passes
  bool tried = false;           // keep has been decided
  double2* keep = nullptr;      // [ns][pts] spectra of the steps, in tile order; null: not kept
  double2* one = nullptr;       // [pts] spectrum of one step, made again
  double* dot = nullptr;        // [pts]
  double* gpart = nullptr;      // [ntiles][3]
  int* frq = nullptr;           // [gx + gy + gz] frequency by position
  int tile = 0, ntiles = 0;
  size_t pts = 0;
  bool kept = false;            // by the last forward pass
};

struct adscf_ctx;
void adj_mx_free(AdjMx* X);
int adj_mx_forward(adscf_ctx* ctx, AdjMx* X);   // chains, spectra where they are kept, and contour integral
// b: [2][npts] cotangents, sc: scalars of the forward pass (device), spec2: [npts] scratch
int adj_mx_backward(adscf_ctx* ctx, AdjMx* X, const double* b, const double* sc, double2* spec2);

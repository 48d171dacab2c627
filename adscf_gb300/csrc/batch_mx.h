// batch_mx.h -- mixed-radix passes of a bulk batch (batch_mx.cu).
#pragma once
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "bulk_kernels.cuh"

struct BatchMx;

// One instance: arrays on the device (T of the batch), natural-order tables on
// the host
struct BatchMxInst {
  int gx, gy, gz, ns;
  const void* inst;             // BulkDev<T> in the batch's array
  void *spec, *slices;
  const void *E, *fk;           // fk: factors of the instance, g_xy first
  const double* g64;
};

// Passes of the instances whose grid has a plan (taken; none in a batch of more
// than 64 grids); null: no memory, err
template <typename T>
BatchMx* batch_mx_create(int dev, const std::vector<BatchMxInst>& in, std::vector<char>& taken, std::string& err);
void batch_mx_destroy(BatchMx* B);
// both chains of every instance taken, on s and the batch's own streams beside it
int batch_mx_enqueue(BatchMx* B, cudaStream_t s, std::string& err);
int batch_mx_launches(const BatchMx* B);

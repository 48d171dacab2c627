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

// null: a grid without a plan, or no memory
template <typename T>
BatchMx* batch_mx_create(int dev, const std::vector<BatchMxInst>& in);
void batch_mx_destroy(BatchMx* B);
// both chains of every instance, on s and the batch's own streams beside it
int batch_mx_enqueue(BatchMx* B, cudaStream_t s, std::string& err);
int batch_mx_launches(const BatchMx* B);

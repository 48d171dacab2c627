// batch_mx.cu -- the chains of a bulk batch on the mixed-radix passes.
//
// Instances of one grid form a class: one launch per pass and step runs all of
// them that are still on their contour (blockIdx.y, instances by descending
// Ns), each with its own factors and arrays.  Classes share nothing and run
// on streams of their own beside each other, so a small class does not wait at
// every step for a large one and the tail of one class's wave is filled by the
// others.
//
// Against the persistent sweep of the line passes (batch.cu), a double step
// reads and writes the spectrum twice for four times and needs no waits
// between items.  An SCF iteration of 64 grids of 24^3 to 64^3, 100 to 200
// steps: split 42.1 -> 23.9 ms, FP64 348 -> 213; of one 64^3 grid 19.1 -> 3.3
// and 153 -> 9.3.
#include <map>
#include <new>
#include <tuple>

#include "batch_mx.h"
#include "bulk_host.h"
#include "bulk_mx_plan.h"

namespace {

// Grids of one batch: each adds a stream and two graph nodes a step, captured on
// the first pass (64 instances of 16^3 to 30^3, 100 steps: 4 grids 4.7 ms an
// iteration and 12.7 ms the first, 64 grids 6.8 and 49; the sweep 68 to 76).  A
// batch of more runs the sweep, whose results differ at rounding.
constexpr size_t kMaxGrids = 64;

struct Class {
  BulkMx M;
  void* d_ios = nullptr;                // Io<T> of the class's instances
  void* d_tab = nullptr;                // their factor tables
  std::vector<int> active;              // instances on their contour at step t
  cudaStream_t st = nullptr;
  cudaEvent_t done = nullptr;
};

}  // namespace

struct BatchMx {
  bool f64 = false;
  std::vector<Class> cls;
  cudaEvent_t fork = nullptr;
};

namespace {

// Plan of a grid, from its sizes alone: an instance's result does not depend on
// what else is in the batch.  FP64 radices as in mx_setup, up to npts / 19456; the
// number of instances with the grid in its place spared large classes a stage
// (64 grids of 32^3 447 us a double step, 466 with this rule) but cost others more
// (64 of 48^3 1926 and 1699, 64 of 24^3 to 64^3 1362 and 1322).  false: lines or
// tiles the passes do not take.
template <typename T>
bool plan_class(Class& C, int optin, int gx, int gy, int gz) {
  BulkMx* M = &C.M;
  const int rmax = sizeof(T) == 4 ? 16 : std::max(5, std::min(16, gx * gy * gz / 19456));
  if (!mx_axis(gx, rmax, M->a[0]) || !mx_axis(gy, rmax, M->a[1]) || !mx_axis(gz, rmax, M->a[2])) return false;
  if (M->a[0].nst + M->a[1].nst > mxk::kMaxSteps || M->a[1].nst + M->a[2].nst > mxk::kMaxSteps) return false;
  M->optin = optin;
  mxk::Dev<T>& D = M->dev<T>();
  D.gx = gx; D.gy = gy; D.gz = gz;
  // 64-byte column runs: 64 grids of 24^3 to 64^3 split 23.9 ms an iteration, 26.7
  // with 32 bytes, 27.3 with 128; the same in FP64
  Geom G;
  if (!default_geometry<T>(M, G)) return false;
  if (!geometry<T>(M, G.cut, 2 * G.cols, G.cap_a, G.cap_b)) geometry<T>(M, G.cut, G.cols, G.cap_a, G.cap_b);
  return true;
}

// Tables and lists of the instances `ids` of one grid, by descending Ns
template <typename T>
bool fill_class(Class& C, bool stream, const std::vector<BatchMxInst>& in, const std::vector<int>& ids) {
  BulkMx* M = &C.M;
  mxk::Dev<T>& D = M->dev<T>();
  const int gx = D.gx, gy = D.gy, gz = D.gz;
  const size_t nxy = (size_t)gx * gy;
  D.stream = stream;
  std::vector<cplx<T>> tw;
  std::vector<std::pair<int, int>> seen;
  D.tw_x = bulkhost::twiddle_offset<T>(gx, tw, seen);
  D.tw_y = bulkhost::twiddle_offset<T>(gy, tw, seen);
  D.tw_z = bulkhost::twiddle_offset<T>(gz, tw, seen);
  const size_t nfk = 2 * nxy + 2 * (size_t)gz, ndc = sizeof(T) == 4 ? (size_t)gz * (gy + 2) : 0;
  const size_t each = (nfk * sizeof(T) + ndc * sizeof(float2) + 15) / 16 * 16;
  if (cudaMalloc(&M->d_tw, tw.size() * sizeof(cplx<T>)) || cudaMalloc(&C.d_tab, each * ids.size()) ||
      cudaMalloc(&C.d_ios, ids.size() * sizeof(mxk::Io<T>)) ||
      cudaStreamCreateWithFlags(&C.st, cudaStreamNonBlocking) ||
      cudaEventCreateWithFlags(&C.done, cudaEventDisableTiming))
    return false;
  std::vector<unsigned char> tab(each * ids.size(), 0);
  std::vector<mxk::Io<T>> ios(ids.size());
  int maxns = 0;
  for (size_t k = 0; k < ids.size(); ++k) {
    const BatchMxInst& q = in[ids[k]];
    unsigned char *h = tab.data() + k * each, *d = static_cast<unsigned char*>(C.d_tab) + k * each;
    const std::vector<T> fk = mx_table<T>(M, static_cast<const T*>(q.fk));
    std::copy(fk.begin(), fk.end(), reinterpret_cast<T*>(h));
    mxk::Io<T>& io = ios[k];
    io.fk = reinterpret_cast<const T*>(d);
    if (sizeof(T) == 4) {
      float2* dc = reinterpret_cast<float2*>(d + nfk * sizeof(T));
      float2* hc = reinterpret_cast<float2*>(h + nfk * sizeof(T)) + (size_t)gz * (gy + 1);
      for (int i = 0; i < gz; ++i) {
        const float hi = (float)q.g64[i];
        hc[i] = make_float2(hi, (float)(q.g64[i] - (double)hi));
      }
      io.dcin = dc;
      io.dcout = dc + (size_t)gz * gy;
      io.dcc = dc + (size_t)gz * (gy + 1);
    }
    io.I = static_cast<const BulkDev<T>*>(q.inst);
    io.spec = static_cast<cplx<T>*>(q.spec);
    io.slices = static_cast<cplx<T>*>(q.slices);
    io.E = static_cast<const T*>(q.E);
    maxns = std::max(maxns, q.ns);
  }
  C.active.assign(maxns + 1, 0);
  for (int id : ids)
    for (int t = 0; t <= in[id].ns; ++t) ++C.active[t];
  D.tw = static_cast<const cplx<T>*>(M->d_tw);
  return !cudaMemcpy(M->d_tw, tw.data(), tw.size() * sizeof(cplx<T>), cudaMemcpyHostToDevice) &&
         !cudaMemcpy(C.d_tab, tab.data(), tab.size(), cudaMemcpyHostToDevice) &&
         !cudaMemcpy(C.d_ios, ios.data(), ios.size() * sizeof(mxk::Io<T>), cudaMemcpyHostToDevice) &&
         !cudaFuncSetAttribute(k_mx_a_b<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin) &&
         !cudaFuncSetAttribute(k_mx_b_b<T, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin) &&
         !cudaFuncSetAttribute(k_mx_b_b<T, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin);
}

template <typename T>
void chains(Class& C) {
  const BulkMx& M = C.M;
  const mxk::Dev<T>& D = C.M.dev<T>();
  const mxk::Io<T>* ios = static_cast<const mxk::Io<T>*>(C.d_ios);
  k_mx_a_b<T><<<dim3(M.grid_a, C.active[0]), M.thr_a, M.sm_a, C.st>>>(D, ios, 0);
  for (int t = 1; t < (int)C.active.size(); ++t) {
    launch<T>(M.thr_b > 256 ? k_mx_b_b<T, 512> : k_mx_b_b<T, 256>, dim3(M.grid_b, C.active[t]), M.thr_b, M.sm_b, C.st,
              D, ios);
    launch<T>(k_mx_a_b<T>, dim3(M.grid_a, C.active[t]), M.thr_a, M.sm_a, C.st, D, ios, t);
  }
}

}  // namespace

template <typename T>
BatchMx* batch_mx_create(int dev, const std::vector<BatchMxInst>& in, std::vector<char>& taken, std::string& err) {
  BatchMx* B = new (std::nothrow) BatchMx();
  if (!B) {
    err = "host memory";
    return nullptr;
  }
  B->f64 = sizeof(T) == 8;
  taken.assign(in.size(), 0);
  std::map<std::tuple<int, int, int>, std::vector<int>> groups;
  for (int i = 0; i < (int)in.size(); ++i) groups[{in[i].gx, in[i].gy, in[i].gz}].push_back(i);
  if (groups.size() > kMaxGrids) return B;
  // factors, spectra and nodes of the batch past L2: stream (as for one large
  // grid: 24.0 against 25.2 ms an iteration of 64 grids)
  size_t pts = 0;
  for (const BatchMxInst& q : in) pts += (size_t)q.gx * q.gy * q.gz;
  int l2 = 0, optin = 0;
  cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
  bool ok = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
            cudaEventCreateWithFlags(&B->fork, cudaEventDisableTiming) == cudaSuccess;
  for (auto& g : groups) {
    Class plan;
    if (!plan_class<T>(plan, optin, std::get<0>(g.first), std::get<1>(g.first), std::get<2>(g.first))) continue;
    std::vector<int>& ids = g.second;
    std::stable_sort(ids.begin(), ids.end(), [&](int a, int b) { return in[a].ns > in[b].ns; });
    for (int i : ids) taken[i] = 1;
    // at most 65535 instances a launch (gridDim.y)
    for (size_t at = 0; at < ids.size() && ok; at += 65535) {
      B->cls.push_back(plan);
      ok = fill_class<T>(B->cls.back(), pts * 32 > (size_t)l2, in,
                         std::vector<int>(ids.begin() + at, ids.begin() + std::min(ids.size(), at + 65535)));
    }
  }
  if (!ok) {
    err = cudaGetErrorString(cudaGetLastError());
    batch_mx_destroy(B);
    return nullptr;
  }
  return B;
}
template BatchMx* batch_mx_create<float>(int, const std::vector<BatchMxInst>&, std::vector<char>&, std::string&);
template BatchMx* batch_mx_create<double>(int, const std::vector<BatchMxInst>&, std::vector<char>&, std::string&);

void batch_mx_destroy(BatchMx* B) {
  if (!B) return;
  for (Class& C : B->cls) {
    cudaFree(C.M.d_tw); cudaFree(C.d_ios); cudaFree(C.d_tab);
    if (C.st) cudaStreamDestroy(C.st);
    if (C.done) cudaEventDestroy(C.done);
  }
  if (B->fork) cudaEventDestroy(B->fork);
  delete B;
}

int batch_mx_enqueue(BatchMx* B, cudaStream_t s, std::string& err) {
  if (B->cls.empty()) return 0;
  cudaError_t e = cudaEventRecord(B->fork, s);
  for (Class& C : B->cls) {
    if (e == cudaSuccess) e = cudaStreamWaitEvent(C.st, B->fork, 0);
    if (e != cudaSuccess) break;
    if (B->f64) chains<double>(C);
    else chains<float>(C);
    e = cudaGetLastError();
    // joined whatever happened: a capture ends only with every stream joined
    cudaEventRecord(C.done, C.st);
    cudaStreamWaitEvent(s, C.done, 0);
  }
  if (e == cudaSuccess) return 0;
  err = cudaGetErrorString(e);
  return 1;
}

// kernel launches of batch_mx_enqueue
int batch_mx_launches(const BatchMx* B) {
  int k = 0;
  for (const Class& C : B->cls) k += 2 * (int)C.active.size() - 1;
  return k;
}

// bulk_mx.cu -- plans, tables, geometry tuner and launches of the mixed-radix
// passes (bulk_mx.cuh).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <tuple>
#include <vector>

#include "bulk_host.h"
#include "bulk_mx_plan.h"
#include "internal.h"

namespace {

template <typename T>
void real_t(adscf_ctx* ctx, int t, bool spread) {
  const BulkMx* M = ctx->mx;
  mxk::Dev<T> D = ctx->mx->dev<T>();
  if constexpr (sizeof(T) == 4) D.io.slices = ctx->hb32.slices;
  else D.io.slices = ctx->hb64.slices;
  D.io.I = static_cast<const BulkDev<T>*>(ctx->d_inst);
  if constexpr (sizeof(T) == 8)
    if (spread) {
      mx_spread_a(D, M->sp, M->grid_a, M->thr_as, M->sm_a, ctx->stream, t);
      return;
    }
  launch<T>(k_mx_a<T>, M->grid_a, M->thr_a, M->sm_a, ctx->stream, D, t);
}
template <typename T>
void step_t(adscf_ctx* ctx, int t) {
  const BulkMx* M = ctx->mx;
  const mxk::Dev<T>& D = ctx->mx->dev<T>();
  if (M->spread) {
    if constexpr (sizeof(T) == 8) mx_spread_b(D, M->sp, M->grid_b, M->thr_bs, M->sm_b, ctx->stream);
  } else {
    launch<T>(M->thr_b > 256 ? k_mx_b<T, 512> : k_mx_b<T, 256>, M->grid_b, M->thr_b, M->sm_b, ctx->stream, D);
  }
  real_t<T>(ctx, t, M->spread);
}

// Geometry tuner, run at context creation on the context's buffers (unit
// Boltzmann factors): the cut first, then columns and threads of k_mx_b, then
// the threads of k_mx_a, each candidate timed as a graph of a few double
// steps, the best of three launches.  How many blocks an SM holds decides, and with
// it how full the last wave is, which no simple rule caught: 160 x 120 x 75
// ran between 32 and 48 us a double step over these choices.  Every geometry
// does the same operations.  Cached per device, grid and precision.
struct GeomKey {
  int dev, gx, gy, gz, prec;
  bool operator<(const GeomKey& o) const {
    return std::tie(dev, gx, gy, gz, prec) < std::tie(o.dev, o.gx, o.gy, o.gz, o.prec);
  }
};
std::mutex g_geom_mu;
std::map<GeomKey, std::pair<Geom, std::string>> g_geom;

template <typename T>
int tune_t(adscf_ctx* ctx) {
  BulkMx* M = ctx->mx;
  const GeomKey key{ctx->dev, ctx->gx, ctx->gy, ctx->gz, ctx->prec};
  {
    std::lock_guard<std::mutex> lk(g_geom_mu);
    auto it = g_geom.find(key);
    if (it != g_geom.end()) {
      const Geom& G = it->second.first;
      geometry<T>(M, G.cut, G.cols, G.cap_a, G.cap_b);
      ctx->tune_report = it->second.second + " (cached)";
      return ADSCF_OK;
    }
  }
  EventPair ev;
  CK(ev.create());
  const int steps = std::min(ctx->ns, ctx->npts > 500000 ? 4 : 16);
  auto time = [&](const Geom& G, float* us) -> int {
    *us = 1e30f;
    if (!geometry<T>(M, G.cut, G.cols, G.cap_a, G.cap_b)) return ADSCF_OK;
    real_t<T>(ctx, 0, M->spread);
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ge = nullptr;
    CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    for (int t = 1; t <= steps; ++t) step_t<T>(ctx, t);
    CK(cudaStreamEndCapture(ctx->stream, &g));
    const cudaError_t ie = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    CK(ie);
    cudaGraphLaunch(ge, ctx->stream);
    for (int round = 0; round < 3; ++round) {
      cudaEventRecord(ev.a, ctx->stream);
      cudaGraphLaunch(ge, ctx->stream);
      cudaEventRecord(ev.b, ctx->stream);
      const cudaError_t se = cudaEventSynchronize(ev.b);
      if (se != cudaSuccess) {
        cudaGraphExecDestroy(ge);
        CK(se);
      }
      float ms = 0.f;
      cudaEventElapsedTime(&ms, ev.a, ev.b);
      *us = std::min(*us, 1000.f * ms / steps);
    }
    cudaGraphExecDestroy(ge);
    return ADSCF_OK;
  };
  Geom best;
  if (!default_geometry<T>(M, best)) return set_err(ctx, ADSCF_E_STATE, "mixed-radix geometry");
  float us = 1e30f;
  int rc;
  auto consider = [&](const Geom& G) -> int {
    float u;
    const int r = time(G, &u);
    if (u < us) { us = u; best = G; }
    return r;
  };
  if ((rc = consider(best))) return rc;
  const Geom start = best;
  for (int k = 0; k <= M->a[1].nst; ++k) {
    Geom G = start;
    G.cut = k;
    const int ro = outer_rows(M, k);
    // a tile 64 times the other one cannot win
    const double r = (double)ro * M->a[0].n / ((double)M->a[1].n / ro * M->a[2].n * G.cols);
    if (k == start.cut || r > 64.0 || r < 1.0 / 64.0) continue;
    if ((rc = consider(G))) return rc;
  }
  const int cut = best.cut;
  for (int cols = 16 / (int)sizeof(cplx<T>); cols <= 128 / (int)sizeof(cplx<T>); cols *= 2)
    for (int cap : {128, 256, 512}) {
      if (cols == start.cols && cap == start.cap_b) continue;
      if (cap > 256 && (M->a[1].n / outer_rows(M, cut)) * M->a[2].n * cols <= 256 * M->a[2].rad[0]) continue;
      if ((rc = consider(Geom{cut, cols, start.cap_a, cap}))) return rc;
    }
  if ((rc = consider(Geom{best.cut, best.cols, 64, best.cap_b}))) return rc;
  if (M->spread && (rc = consider(Geom{best.cut, best.cols, 32, best.cap_b}))) return rc;
  CK(cudaGetLastError());
  geometry<T>(M, best.cut, best.cols, best.cap_a, best.cap_b);
  const mxk::Dev<T>& D = M->dev<T>();
  char line[160];
  std::snprintf(line, sizeof(line),
                "mixed radix %.2f us/double step: row sets of %d, row blocks of %d x %d columns, threads %d and %d", us,
                D.ro, D.mi, D.cols, M->spread ? M->thr_as : M->thr_a, M->spread ? M->thr_bs : M->thr_b);
  ctx->tune_report = line;
  std::lock_guard<std::mutex> lk(g_geom_mu);
  g_geom[key] = {best, line};
  return ADSCF_OK;
}

}  // namespace

// new diffusion factors
template <typename T>
int mx_factors(adscf_ctx* ctx, const std::vector<T>& fk, const std::vector<double>& g64) {
  BulkMx* M = ctx->mx;
  const int gz = ctx->gz;
  std::vector<T> out;
  if (M->yz) {   // g_xy g_z of the rows, and a z axis of one point
    const size_t gx = ctx->gx, nxy = gx * gz;
    std::vector<T> f(2 * nxy + 2, (T)0);
    for (size_t z = 0; z < (size_t)gz; ++z)
      for (size_t x = 0; x < gx; ++x) f[z * gx + x] = fk[x] * fk[2 * gx + z];
    f[2 * nxy] = (T)1;
    out = mx_table<T>(M, f.data());
  } else {
    out = mx_table<T>(M, fk.data());
  }
  CK(cudaMemcpy(M->d_fk, out.data(), out.size() * sizeof(T), cudaMemcpyHostToDevice));
  if (sizeof(T) == 4) {
    std::vector<float2> c(gz);
    for (int i = 0; i < gz; ++i) {
      const float h = (float)g64[i];
      c[i] = make_float2(h, (float)(g64[i] - (double)h));
    }
    CK(cudaMemcpy(const_cast<float2*>(M->dev<T>().io.dcc), c.data(), gz * sizeof(float2), cudaMemcpyHostToDevice));
  }
  return ADSCF_OK;
}

template int mx_factors<float>(adscf_ctx*, const std::vector<float>&, const std::vector<double>&);
template int mx_factors<double>(adscf_ctx*, const std::vector<double>&, const std::vector<double>&);

// Plans and tables.  FP32 radices go up to 16: the fewest stages.  FP64:
// npts / 19456 (the 608 SM quarters times 32 lanes), 5 at least: with fewer
// butterflies than lanes a larger radix only lengthens each quarter's
// program.  A grid whose lines do not fit leaves ctx->mx null (the generic
// passes run it).
template <typename T>
int mx_setup(adscf_ctx* ctx, const BulkDev<T>& I, const std::vector<T>& fk, const std::vector<double>& g64) {
  BulkMx* M = new (std::nothrow) BulkMx();
  if (!M) return set_err(ctx, ADSCF_E_OOM, "mixed-radix plan");
  const int rmax = sizeof(T) == 4 ? 16 : std::max(5, std::min(16, ctx->npts / 19456));
  Geom G;
  mxk::Dev<T>& D = M->dev<T>();
  auto plan = [&](int gx, int gy, int gz) {
    D.gx = gx; D.gy = gy; D.gz = gz;
    return mx_axis(gx, rmax, M->a[0]) && mx_axis(gy, rmax, M->a[1]) && mx_axis(gz, rmax, M->a[2]) &&
           M->a[0].nst + M->a[1].nst <= mxk::kMaxSteps && M->a[1].nst + M->a[2].nst <= mxk::kMaxSteps &&
           default_geometry<T>(M, G);
  };
  bool ok = cudaDeviceGetAttribute(&M->optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->dev) == cudaSuccess;
  // FP64 grids of one y row take z for y, the axis that is cut between the
  // passes: a block then holds 100 of the 300 points of a z line of 64 x 1 x 300
  // (27.0 and 26.4 us a double step, 21.7 with an output per lane).  FP32 keeps
  // its (0, 0) pencil along z.
  M->yz = sizeof(T) == 8 && ctx->gy == 1 && ctx->gz > 1 && ok && plan(ctx->gx, ctx->gz, 1);
  if (!M->yz) ok = ok && plan(ctx->gx, ctx->gy, ctx->gz);
  const int gx = D.gx, gy = D.gy, gz = D.gz;
  // Where the factors, spectrum and node (32 bytes a point) exceed L2, factors
  // and nodes stream so that the spectrum stays: 256^3 362 -> 352 us a double
  // step, 160^3 98 -> 93, 128 x 128 x 256 92 -> 85; below, the factors stay too
  // (64 x 64 x 256 27.7 us, 29.3 streamed).
  int l2 = 0;
  if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, ctx->dev) == cudaSuccess) D.stream = (size_t)ctx->npts * 32 > (size_t)l2;
  if (!ok) {
    delete M;
    return ADSCF_OK;
  }
  ctx->mx = M;
  if (sizeof(T) == 8) {
    // An output per lane up to 32768 points, whose radix-4 stages are 256 warps
    // of butterflies on 608 SM quarters: us a double step without and with,
    // 16^3 20.1 and 12.8, 32 x 1 x 64 18.6 and 13.4, 64 x 1 x 300 26.8 and 21.7,
    // 24^3 21.0 and 18.0, 32^3 22.8 and 21.8; above, the quarters have work
    // enough and the repeated additions cost more (40^3 37.3 and 51.2).
    M->spread = ctx->npts <= 32768;
    for (const mxk::Axis& A : M->a)
      for (int i = 0; i < A.nst; ++i) M->spread = M->spread && A.rad[i] <= 5;
    CK(mx_spread_setup(M->optin));
  }
  CK(cudaFuncSetAttribute(k_mx_a<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin));
  CK(cudaFuncSetAttribute(k_mx_b<T, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin));
  CK(cudaFuncSetAttribute(k_mx_b<T, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin));
  std::vector<cplx<T>> tw;
  std::vector<std::pair<int, int>> seen;
  D.tw_x = bulkhost::twiddle_offset<T>(gx, tw, seen);
  D.tw_y = bulkhost::twiddle_offset<T>(gy, tw, seen);
  D.tw_z = bulkhost::twiddle_offset<T>(gz, tw, seen);
  // one allocation: twiddles, factors, the pencil's rows
  const size_t twb = (tw.size() * sizeof(cplx<T>) + 255) / 256 * 256;
  const size_t fkb = ((2 * (size_t)gx * gy + 2 * (size_t)gz) * sizeof(T) + 255) / 256 * 256;
  const size_t dcb = sizeof(T) == 4 ? (size_t)gz * (gy + 2) * sizeof(float2) : 0;
  CK(cudaMalloc(&M->d_tw, twb + fkb + dcb));
  CK(cudaMemcpy(M->d_tw, tw.data(), tw.size() * sizeof(cplx<T>), cudaMemcpyHostToDevice));
  M->d_fk = static_cast<unsigned char*>(M->d_tw) + twb;
  if (sizeof(T) == 4) {
    float2* dc = reinterpret_cast<float2*>(static_cast<unsigned char*>(M->d_fk) + fkb);
    CK(cudaMemset(dc, 0, dcb));
    D.io.dcin = dc;
    D.io.dcout = dc + (size_t)gz * gy;
    D.io.dcc = D.io.dcout + gz;
  }
  D.tw = static_cast<const cplx<T>*>(M->d_tw);
  D.io.fk = static_cast<const T*>(M->d_fk);
  D.io.spec = I.spec;
  D.io.E = I.E;
  return mx_factors<T>(ctx, fk, g64);
}
template int mx_setup<float>(adscf_ctx*, const BulkDev<float>&, const std::vector<float>&, const std::vector<double>&);
template int mx_setup<double>(adscf_ctx*, const BulkDev<double>&, const std::vector<double>&, const std::vector<double>&);

void mx_destroy(adscf_ctx* ctx) {
  if (!ctx->mx) return;
  cudaFree(ctx->mx->d_tw);
  delete ctx->mx;
  ctx->mx = nullptr;
}

// real-space pass of node t, and a whole double step
void mx_real(adscf_ctx* ctx, int t) {
  if (ctx->prec == ADSCF_SPLIT) real_t<float>(ctx, t, false);
  else real_t<double>(ctx, t, ctx->mx->spread);
}
void mx_step(adscf_ctx* ctx, int t) {
  if (ctx->prec == ADSCF_SPLIT) step_t<float>(ctx, t);
  else step_t<double>(ctx, t);
}
int mx_tune(adscf_ctx* ctx) { return ctx->prec == ADSCF_SPLIT ? tune_t<float>(ctx) : tune_t<double>(ctx); }

bool mx_launch64(const adscf_ctx* ctx, MxLaunch64& L) {
  const BulkMx* M = ctx->mx;
  if (!M || ctx->prec != ADSCF_FP64) return false;
  L = MxLaunch64{M->d64, M->yz, M->thr_a, M->thr_b, M->grid_a, M->grid_b, M->sm_a, M->sm_b, M->optin,
                 M->spread, M->sp, M->thr_as, M->thr_bs};
  L.D.io.slices = ctx->hb64.slices;
  L.D.io.I = static_cast<const BulkDev<double>*>(ctx->d_inst);
  return true;
}
void mx_freqs(const adscf_ctx* ctx, std::vector<int>& f) {
  f.clear();
  for (const mxk::Axis& A : ctx->mx->a)
    for (int p = 0; p < A.n; ++p) f.push_back(mx_freq(A, p));
}

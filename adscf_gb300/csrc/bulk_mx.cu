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
#include "bulk_mx.cuh"
#include "internal.h"
#include "launch_pdl.h"

// Launch geometry and tables of the mixed-radix passes of one context.
struct BulkMx {
  mxk::Axis a[3];               // x, y, z
  int thr_a = 32, thr_b = 32, grid_a = 0, grid_b = 0;
  size_t sm_a = 0, sm_b = 0;
  void* d_tw = nullptr;         // twiddles (cplx<T>)
  void* d_fk = nullptr;         // diffusion factors by position (T)
  float2* d_dc = nullptr;       // dcin [gz][gy], dcout [gz], kernel [gz]
  int optin = 0;                // opt-in shared memory per block
  template <typename T> mxk::Dev<T>& dev();
  mxk::Dev<float> d32{};
  mxk::Dev<double> d64{};
};
template <> mxk::Dev<float>& BulkMx::dev<float>() { return d32; }
template <> mxk::Dev<double>& BulkMx::dev<double>() { return d64; }

namespace {

// ---- mixed-radix passes (bulk_mx.cuh) ---------------------------------------
// Radices of an n-point line, at most rmax each (at least 5): the fewest
// stages, then the smallest largest radix; the largest comes last, where it
// needs no twiddles.
bool mx_axis(int n, int rmax, mxk::Axis& A) {
  static const int kRad[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
  A = mxk::Axis{};
  A.n = n;
  std::vector<int> best, cur;
  auto better = [&](const std::vector<int>& c) {
    if (best.empty()) return true;
    if (c.size() != best.size()) return c.size() < best.size();
    return *std::max_element(c.begin(), c.end()) < *std::max_element(best.begin(), best.end());
  };
  auto dfs = [&](auto&& self, int m, int cap) -> void {
    if (m == 1) {
      if (better(cur)) best = cur;
      return;
    }
    if ((int)cur.size() == mxk::kMaxStages) return;
    for (int r : kRad)
      if (r <= cap && m % r == 0) {
        cur.push_back(r);
        self(self, m / r, r);
        cur.pop_back();
      }
  };
  if (n > 1024) return false;
  if (n > 1) {
    dfs(dfs, n, std::max(5, rmax));
    if (best.empty()) return false;
  }
  std::sort(best.begin(), best.end());
  A.nst = (int)best.size();
  int m = n;
  for (int i = 0; i < A.nst; ++i) {
    A.rad[i] = best[i];
    A.m[i] = m;
    m /= best[i];
  }
  return true;
}
// frequency of position p of a line
int mx_freq(const mxk::Axis& A, int p) {
  int k = 0, f = 1, m = A.n;
  for (int i = 0; i < A.nst; ++i) {
    m /= A.rad[i];
    k += f * (p / m);
    p %= m;
    f *= A.rad[i];
  }
  return k;
}

// Row pitch of k_mx_b's tile: an odd number of columns, so that the rows of a z
// stage's lines lie in different banks (256^3 split 409 -> 362 us a double step,
// 128 x 128 x 256 106 -> 92, 60 x 72 x 100 18.7 -> 17.9).
int pitch_b(int gz, int mi, int cols) { return (mi > 1 ? gz | 1 : gz) * cols; }

template <typename T>
size_t bytes_a(const BulkMx* M, int ro) {
  return ((size_t)ro * (M->a[0].n | 1) + M->a[0].n + M->a[1].n) * sizeof(cplx<T>);
}
template <typename T>
size_t bytes_b(const BulkMx* M, int mi, int cols) {
  const size_t gy = M->a[1].n, gz = M->a[2].n;
  const size_t tile = (mi * pitch_b((int)gz, mi, cols) + gy + gz) * sizeof(cplx<T>) + 2 * gz * sizeof(T);
  return sizeof(T) == 4 ? std::max(tile, 2 * (gz + 1) * sizeof(float2) + 8 * gz * sizeof(float4)) : tile;
}
int outer_rows(const BulkMx* M, int cut) {
  int ro = 1;
  for (int i = 0; i < cut; ++i) ro *= M->a[1].rad[i];
  return ro;
}

// Geometry: the y cut, k_mx_b's columns and the threads of both kernels.
// Fills the tile sizes and step programs; false if a tile does not fit.
template <typename T>
bool geometry(BulkMx* M, int cut, int cols, int cap_a, int cap_b) {
  const mxk::Axis &X = M->a[0], &Y = M->a[1], &Z = M->a[2];
  mxk::Dev<T>& D = M->dev<T>();
  const int gx = X.n, gy = Y.n, gz = Z.n;
  const int ro = outer_rows(M, cut), mi = gy / ro, pitch = gx | 1;
  if (bytes_a<T>(M, ro) > (size_t)M->optin || bytes_b<T>(M, mi, cols) > (size_t)M->optin) return false;
  D.ro = ro; D.mi = mi;
  D.pitch = pitch;
  D.cols = cols;
  for (D.lc = 0; (1 << D.lc) < cols;) ++D.lc;
  D.pb = pitch_b(gz, mi, cols);
  D.ctiles = (gx + cols - 1) / cols;
  D.ntiles = D.ctiles * ro;
  D.rx = X.nst ? X.rad[0] : 1;
  D.rz = Z.nst ? Z.rad[Z.nst - 1] : 1;
  D.nxs = X.nst > 1 ? X.nst - 1 : 0;
  D.mgj = mxk::div_magic(gx / D.rx);
  D.mgz = mxk::div_magic(mi << D.lc);
  D.a.n = D.b.n = 0;
  auto step = [&](const mxk::Axis& A, int s, int scale, int npts, int lines) {
    mxk::Step S{};
    S.R = A.rad[s];
    S.m = A.m[s] / scale;
    S.mp = S.m / S.R;
    S.lines = lines;
    S.total = npts / S.R * lines;
    S.mg = (1u << 20) / (unsigned)S.mp + 1;
    S.mgl = mxk::div_magic(lines);
    S.lmask = 0x7fffffff; S.lsh = 31;
    S.tws = A.n / A.m[s];
    S.jmul = scale; S.jin = scale > 1 ? 1 : 0;
    return S;
  };
  for (int s = 1; s < X.nst; ++s) {           // k_mx_a: lines are the tile's rows
    mxk::Step S = step(X, s, 1, gx, ro);
    S.ls = pitch; S.es = 1;
    S.gls = 0; S.ges = 1;                     // in or out directly only where a tile is one row
    S.tw = ro * pitch;
    D.a.s[D.a.n++] = S;
  }
  for (int s = 0; s < cut; ++s) {             // outer y stages: lines x, rows M' apart
    mxk::Step S = step(Y, s, mi, ro, gx);
    S.ls = 1; S.es = pitch;
    S.gls = 1; S.ges = mi * gx;
    S.tw = ro * pitch + gx;
    D.a.s[D.a.n++] = S;
  }
  const int pts = mi * D.pb;                  // k_mx_b: tile [y'][z][c]
  for (int s = cut; s < Y.nst; ++s) {         // inner y stages: lines (z, c)
    mxk::Step S = step(Y, s, 1, mi, gz << D.lc);
    S.lmask = cols - 1; S.lsh = D.lc;
    S.ls = 1; S.ls2 = cols; S.es = D.pb;
    S.gls = 1; S.gls2 = gx * gy; S.ges = gx;
    S.tw = pts;
    D.b.s[D.b.n++] = S;
  }
  for (int s = 0; s + 1 < Z.nst; ++s) {       // z stages: lines (y', c)
    mxk::Step S = step(Z, s, 1, gz, mi << D.lc);
    S.lmask = cols - 1; S.lsh = D.lc;
    S.ls = 1; S.ls2 = D.pb; S.es = cols;
    S.gls = 1; S.gls2 = gx; S.ges = gx * gy;
    S.tw = pts + gy;
    D.b.s[D.b.n++] = S;
  }
  int max_a = gx / D.rx * ro, max_b = gz / D.rz * (mi << D.lc);
  for (int i = 0; i < D.a.n; ++i) max_a = std::max(max_a, D.a.s[i].total);
  for (int i = 0; i < D.b.n; ++i) max_b = std::max(max_b, D.b.s[i].total);
  auto threads = [](int tasks, int cap) { return std::min(cap, std::max(32, (tasks + 31) / 32 * 32)); };
  M->thr_a = threads(max_a, cap_a);
  M->thr_b = threads(max_b, cap_b);
  M->grid_a = mi * gz;
  M->grid_b = D.ntiles;
  if (sizeof(T) == 4) M->grid_b += (gz + M->thr_b / 32 - 1) / (M->thr_b / 32);
  M->sm_a = bytes_a<T>(M, ro);
  M->sm_b = bytes_b<T>(M, mi, cols);
  return true;
}

struct Geom {
  int cut, cols, cap_a, cap_b;
};
// Without the tuner: 32-byte column runs, and the cut that brings the two
// tiles' sizes closest
template <typename T>
bool default_geometry(BulkMx* M, Geom& G) {
  G = Geom{-1, 32 / (int)sizeof(cplx<T>), 128, 256};
  double best = 1e300;
  for (int k = 0; k <= M->a[1].nst; ++k) {
    const int ro = outer_rows(M, k), mi = M->a[1].n / ro;
    const double cost = std::fabs(std::log((double)ro * M->a[0].n / ((double)mi * M->a[2].n * G.cols)));
    if (cost < best && geometry<T>(M, k, G.cols, G.cap_a, G.cap_b)) { best = cost; G.cut = k; }
  }
  if (G.cut < 0) {
    G.cols = 1;
    for (int k = 0; k <= M->a[1].nst && G.cut < 0; ++k)
      if (geometry<T>(M, k, 1, G.cap_a, G.cap_b)) G.cut = k;
  }
  return G.cut >= 0 && geometry<T>(M, G.cut, G.cols, G.cap_a, G.cap_b);
}

// FP32 passes are launched programmatically (the next pass's blocks start and
// load their tables while the last ones of this pass run: 25 x 27 x 30 12.8 ->
// 11.0 us a double step).  FP64 passes are not: blocks that wait early take
// the places of FP64 blocks that could work, which then share the FP64 pipes
// of fewer SMs (48^3 60 us with, 43 us without; 32^3 32 and 23).
template <typename T, typename... KArgs, typename... Args>
void launch(void (*kern)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, Args&&... args) {
  if constexpr (sizeof(T) == 4) launch_pdl(kern, grid, block, smem, s, std::forward<Args>(args)...);
  else kern<<<grid, block, smem, s>>>(args...);
}
template <typename T>
void real_t(adscf_ctx* ctx, int t) {
  const BulkMx* M = ctx->mx;
  mxk::Dev<T> D = ctx->mx->dev<T>();
  if constexpr (sizeof(T) == 4) D.slices = ctx->hb32.slices;
  else D.slices = ctx->hb64.slices;
  D.I = static_cast<const BulkDev<T>*>(ctx->d_inst);
  launch<T>(k_mx_a<T>, M->grid_a, M->thr_a, M->sm_a, ctx->stream, D, t);
}
template <typename T>
void step_t(adscf_ctx* ctx, int t) {
  const BulkMx* M = ctx->mx;
  const mxk::Dev<T>& D = ctx->mx->dev<T>();
  launch<T>(M->thr_b > 256 ? k_mx_b<T, 512> : k_mx_b<T, 256>, M->grid_b, M->thr_b, M->sm_b, ctx->stream, D);
  real_t<T>(ctx, t);
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
    real_t<T>(ctx, 0);
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
  CK(cudaGetLastError());
  geometry<T>(M, best.cut, best.cols, best.cap_a, best.cap_b);
  const mxk::Dev<T>& D = M->dev<T>();
  char line[160];
  std::snprintf(line, sizeof(line),
                "mixed radix %.2f us/double step: row sets of %d, row blocks of %d x %d columns, threads %d and %d", us,
                D.ro, D.mi, D.cols, M->thr_a, M->thr_b);
  ctx->tune_report = line;
  std::lock_guard<std::mutex> lk(g_geom_mu);
  g_geom[key] = {best, line};
  return ADSCF_OK;
}

}  // namespace

// diffusion factors by position, from the natural-order tables of
// append_tables; FP32: none for the (0, 0) pencil, which has its own blocks
template <typename T>
int mx_factors(adscf_ctx* ctx, const std::vector<T>& fk, const std::vector<double>& g64) {
  BulkMx* M = ctx->mx;
  const int gx = ctx->gx, gy = ctx->gy, gz = ctx->gz;
  const size_t nxy = (size_t)gx * gy;
  std::vector<T> out(2 * nxy + 2 * (size_t)gz);
  std::vector<int> f[3];
  for (int d = 0; d < 3; ++d)
    for (int p = 0; p < M->a[d].n; ++p) f[d].push_back(mx_freq(M->a[d], p));
  for (int h = 0; h < 2; ++h) {
    for (int y = 0; y < gy; ++y) {
      const T* from = fk.data() + h * nxy + (size_t)f[1][y] * gx;
      T* to = out.data() + h * nxy + (size_t)y * gx;
      for (int x = 0; x < gx; ++x) to[x] = from[f[0][x]];
    }
    for (int z = 0; z < gz; ++z) out[2 * nxy + (size_t)h * gz + z] = fk[2 * nxy + (size_t)h * gz + f[2][z]];
  }
  if (sizeof(T) == 4) out[0] = out[nxy] = (T)0;
  CK(cudaMemcpy(M->d_fk, out.data(), out.size() * sizeof(T), cudaMemcpyHostToDevice));
  if (sizeof(T) == 4) {
    std::vector<float2> c(gz);
    for (int i = 0; i < gz; ++i) {
      const float h = (float)g64[i];
      c[i] = make_float2(h, (float)(g64[i] - (double)h));
    }
    CK(cudaMemcpy(const_cast<float2*>(M->dev<T>().dcc), c.data(), gz * sizeof(float2), cudaMemcpyHostToDevice));
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
  const int gx = ctx->gx, gy = ctx->gy, gz = ctx->gz;
  const int rmax = sizeof(T) == 4 ? 16 : std::max(5, std::min(16, ctx->npts / 19456));
  Geom G;
  const bool ok = mx_axis(gx, rmax, M->a[0]) && mx_axis(gy, rmax, M->a[1]) && mx_axis(gz, rmax, M->a[2]) &&
                  M->a[0].nst + M->a[1].nst <= mxk::kMaxSteps && M->a[1].nst + M->a[2].nst <= mxk::kMaxSteps &&
                  cudaDeviceGetAttribute(&M->optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->dev) == cudaSuccess;
  mxk::Dev<T>& D = M->dev<T>();
  D.gx = gx; D.gy = gy; D.gz = gz;
  // Where the factors, spectrum and node (32 bytes a point) exceed L2, factors
  // and nodes stream so that the spectrum stays: 256^3 362 -> 352 us a double
  // step, 160^3 98 -> 93, 128 x 128 x 256 92 -> 85; below, the factors stay too
  // (64 x 64 x 256 27.7 us, 29.3 streamed).
  int l2 = 0;
  if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, ctx->dev) == cudaSuccess) D.stream = (size_t)ctx->npts * 32 > (size_t)l2;
  if (!ok || !default_geometry<T>(M, G)) {
    delete M;
    return ADSCF_OK;
  }
  ctx->mx = M;
  CK(cudaFuncSetAttribute(k_mx_a<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin));
  CK(cudaFuncSetAttribute(k_mx_b<T, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin));
  CK(cudaFuncSetAttribute(k_mx_b<T, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, M->optin));
  std::vector<cplx<T>> tw;
  std::vector<std::pair<int, int>> seen;
  D.tw_x = bulkhost::twiddle_offset<T>(gx, tw, seen);
  D.tw_y = bulkhost::twiddle_offset<T>(gy, tw, seen);
  D.tw_z = bulkhost::twiddle_offset<T>(gz, tw, seen);
  CK(cudaMalloc(&M->d_tw, tw.size() * sizeof(cplx<T>)));
  CK(cudaMemcpy(M->d_tw, tw.data(), tw.size() * sizeof(cplx<T>), cudaMemcpyHostToDevice));
  CK(cudaMalloc(&M->d_fk, (2 * (size_t)gx * gy + 2 * (size_t)gz) * sizeof(T)));
  if (sizeof(T) == 4) {
    const size_t n = (size_t)gz * (gy + 2);
    CK(cudaMalloc(&M->d_dc, n * sizeof(float2)));
    CK(cudaMemset(M->d_dc, 0, n * sizeof(float2)));
    D.dcin = M->d_dc;
    D.dcout = M->d_dc + (size_t)gz * gy;
    D.dcc = D.dcout + gz;
  }
  D.tw = static_cast<const cplx<T>*>(M->d_tw);
  D.fk = static_cast<const T*>(M->d_fk);
  D.spec = I.spec;
  D.E = I.E;
  return mx_factors<T>(ctx, fk, g64);
}
template int mx_setup<float>(adscf_ctx*, const BulkDev<float>&, const std::vector<float>&, const std::vector<double>&);
template int mx_setup<double>(adscf_ctx*, const BulkDev<double>&, const std::vector<double>&, const std::vector<double>&);

void mx_destroy(adscf_ctx* ctx) {
  if (!ctx->mx) return;
  cudaFree(ctx->mx->d_tw);
  cudaFree(ctx->mx->d_fk);
  cudaFree(ctx->mx->d_dc);
  delete ctx->mx;
  ctx->mx = nullptr;
}

// real-space pass of node t, and a whole double step
void mx_real(adscf_ctx* ctx, int t) {
  if (ctx->prec == ADSCF_SPLIT) real_t<float>(ctx, t);
  else real_t<double>(ctx, t);
}
void mx_step(adscf_ctx* ctx, int t) {
  if (ctx->prec == ADSCF_SPLIT) step_t<float>(ctx, t);
  else step_t<double>(ctx, t);
}
int mx_tune(adscf_ctx* ctx) { return ctx->prec == ADSCF_SPLIT ? tune_t<float>(ctx) : tune_t<double>(ctx); }

bool mx_launch64(const adscf_ctx* ctx, MxLaunch64& L) {
  const BulkMx* M = ctx->mx;
  if (!M || ctx->mx_off || ctx->prec != ADSCF_FP64) return false;
  L = MxLaunch64{M->d64, M->thr_a, M->thr_b, M->grid_a, M->grid_b, M->sm_a, M->sm_b, M->optin};
  L.D.slices = ctx->hb64.slices;
  L.D.I = static_cast<const BulkDev<double>*>(ctx->d_inst);
  return true;
}
void mx_freqs(const adscf_ctx* ctx, std::vector<int>& f) {
  f.clear();
  for (const mxk::Axis& A : ctx->mx->a)
    for (int p = 0; p < A.n; ++p) f.push_back(mx_freq(A, p));
}

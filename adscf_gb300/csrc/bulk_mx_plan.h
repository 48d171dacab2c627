// bulk_mx_plan.h -- plans and launch geometry of the mixed-radix passes
// (bulk_mx.cuh).
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

#include "bulk_mx.cuh"
#include "launch_pdl.h"

// Launch geometry and tables of the mixed-radix passes of one context.
struct BulkMx {
  mxk::Axis a[3];               // x, y, z
  int thr_a = 32, thr_b = 32, grid_a = 0, grid_b = 0;
  int thr_as = 32, thr_bs = 32; // threads of the kernels with an output per lane
  bool spread = false;          // those run the chains
  mxk::Spread sp{};             // and what their inverse stages need
  size_t sm_a = 0, sm_b = 0;
  void* d_tw = nullptr;         // twiddles (cplx<T>), the allocation that holds d_fk too
  void* d_fk = nullptr;         // diffusion factors by position (T)
  int optin = 0;                // opt-in shared memory per block
  bool yz = false;              // the grid's z axis is the passes' y axis
  template <typename T> mxk::Dev<T>& dev();
  mxk::Dev<float> d32{};
  mxk::Dev<double> d64{};
};
template <> inline mxk::Dev<float>& BulkMx::dev<float>() { return d32; }
template <> inline mxk::Dev<double>& BulkMx::dev<double>() { return d64; }

// kernels with an output per lane (bulk_mx_spread.cu), in a file of their own:
// beside those of bulk_mx.cuh they cost the latter 3 % (60 x 72 x 100 split 18.4
// us a double step, 17.9 without)
cudaError_t mx_spread_setup(int optin);
void mx_spread_a(const mxk::Dev<double>& D, const mxk::Spread& W, int grid, int threads, size_t smem, cudaStream_t s,
                 int t);
void mx_spread_b(const mxk::Dev<double>& D, const mxk::Spread& W, int grid, int threads, size_t smem, cudaStream_t s);

namespace {

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

// diffusion factors by position, from the natural-order table fk of
// append_tables; FP32: none for the (0, 0) pencil, which has its own blocks
template <typename T>
std::vector<T> mx_table(const BulkMx* M, const T* fk) {
  const int gx = M->a[0].n, gy = M->a[1].n, gz = M->a[2].n;
  const size_t nxy = (size_t)gx * gy;
  std::vector<T> out(2 * nxy + 2 * (size_t)gz);
  std::vector<int> f[3];
  for (int d = 0; d < 3; ++d)
    for (int p = 0; p < M->a[d].n; ++p) f[d].push_back(mx_freq(M->a[d], p));
  for (int h = 0; h < 2; ++h) {
    for (int y = 0; y < gy; ++y) {
      const T* from = fk + h * nxy + (size_t)f[1][y] * gx;
      T* to = out.data() + h * nxy + (size_t)y * gx;
      for (int x = 0; x < gx; ++x) to[x] = from[f[0][x]];
    }
    for (int z = 0; z < gz; ++z) out[2 * nxy + (size_t)h * gz + z] = fk[2 * nxy + (size_t)h * gz + f[2][z]];
  }
  if (sizeof(T) == 4) out[0] = out[nxy] = (T)0;
  return out;
}

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
  mxk::Spread& W = M->sp;
  W.zrp = Z.nst > 1 ? Z.rad[Z.nst - 2] : 0;
  W.ztwp = Z.nst > 1 ? gz / Z.m[Z.nst - 2] : 0;
  auto prev = [](const mxk::Axis& A, int s, int npts, int m) {
    return s > 0 ? mxk::Prev{A.rad[s - 1], A.n / A.m[s - 1], npts / m} : mxk::Prev{0, 0, 0};
  };
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
    W.a[D.a.n] = prev(X, s, gx, S.m);
    D.a.s[D.a.n++] = S;
  }
  for (int s = 0; s < cut; ++s) {             // outer y stages: lines x, rows M' apart
    mxk::Step S = step(Y, s, mi, ro, gx);
    S.ls = 1; S.es = pitch;
    S.gls = 1; S.ges = mi * gx;
    S.tw = ro * pitch + gx;
    W.a[D.a.n] = prev(Y, s, ro, S.m);
    D.a.s[D.a.n++] = S;
  }
  const int pts = mi * D.pb;                  // k_mx_b: tile [y'][z][c]
  for (int s = cut; s < Y.nst; ++s) {         // inner y stages: lines (z, c)
    mxk::Step S = step(Y, s, 1, mi, gz << D.lc);
    S.lmask = cols - 1; S.lsh = D.lc;
    S.ls = 1; S.ls2 = cols; S.es = D.pb;
    S.gls = 1; S.gls2 = gx * gy; S.ges = gx;
    S.tw = pts;
    W.b[D.b.n] = prev(Y, s, mi, S.m);
    D.b.s[D.b.n++] = S;
  }
  for (int s = 0; s + 1 < Z.nst; ++s) {       // z stages: lines (y', c)
    mxk::Step S = step(Z, s, 1, gz, mi << D.lc);
    S.lmask = cols - 1; S.lsh = D.lc;
    S.ls = 1; S.ls2 = D.pb; S.es = cols;
    S.gls = 1; S.gls2 = gx; S.ges = gx * gy;
    S.tw = pts + gy;
    W.b[D.b.n] = prev(Z, s, gz, S.m);
    D.b.s[D.b.n++] = S;
  }
  int max_a = gx / D.rx * ro, max_b = gz / D.rz * (mi << D.lc);
  for (int i = 0; i < D.a.n; ++i) max_a = std::max(max_a, D.a.s[i].total);
  for (int i = 0; i < D.b.n; ++i) max_b = std::max(max_b, D.b.s[i].total);
  auto threads = [](int tasks, int cap) { return std::min(cap, std::max(32, (tasks + 31) / 32 * 32)); };
  M->thr_a = threads(max_a, cap_a);
  M->thr_b = threads(max_b, cap_b);
  // a lane per output: 32 / R butterflies a warp
  auto warps = [](int tasks, int R) { return (tasks + 32 / R - 1) / (32 / R); };
  int wa = X.nst ? warps(gx / D.rx * ro, D.rx) : 1, wb = Z.nst ? warps(gz / D.rz * (mi << D.lc), D.rz) : 1;
  for (int i = 0; i < D.a.n; ++i) wa = std::max(wa, warps(D.a.s[i].total, D.a.s[i].R));
  for (int i = 0; i < D.b.n; ++i) wb = std::max(wb, warps(D.b.s[i].total, D.b.s[i].R));
  M->thr_as = std::min(2 * cap_a, 32 * wa);
  M->thr_bs = std::min(std::min(256, cap_b), 32 * wb);
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
void launch(void (*kern)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t s, Args&&... args) {
  if constexpr (sizeof(T) == 4) launch_pdl(kern, grid, block, smem, s, std::forward<Args>(args)...);
  else kern<<<grid, block, smem, s>>>(args...);
}
}  // namespace

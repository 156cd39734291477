// Reduced normal system of SDPX's LP standard form and of Lorentz cones
// (include/sdpx_b200_normal.h).
//
// Layout.  B (n × m_eq, column-major, one column per equality) stays resident;
// the scaled operand B̂ has the same layout, so Q = B̂ᵀB̂ is one lower SYRK of
// the FP64 tile engine with the variables as the contraction index:
//   rows [0, n_lp)         B̂ = D^{-1/2} B           (LP, src/lp_solver.jl:1892-1915)
//   rows of cone k         B̂ = W_k⁻¹ B_k            (Lorentz, W_k symmetric, so
//                                                    B̂_kᵀB̂_k = B_kᵀ Hs_k⁻¹ B_k)
// Using W⁻¹ rather than the signed form Hs⁻¹ = (2Jw(Jw)ᵀ − J)/η² keeps the
// contraction a plain positive Gram matrix (no cancellation between a
// rank-one and a diagonal term).
//
// This translation unit is compiled with FMA contraction off (--fmad=false):
// the per-cone kernels then evaluate the reference's scalar recurrences with
// exactly its roundings (IEEE division and square root are correctly rounded),
// so NT scaling points, λ, η, the NT maps and the LP pack are bit-identical to
// a sequential IEEE evaluation in the reference's order.
#include <cuda_runtime.h>

#include <array>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/sdpx_b200_normal.h"
#include "ipm_controller.h"
#include "blas_f64.h"
#include "chol.h"
#include "dbuf.h"
#include "schur_bf16.h"
#include "vec_kernels.h"

namespace sdpx {
namespace {

// A cone's vectors are worked on by a group of g lanes (a power of two up to a warp,
// chosen from the mean dimension): the elementwise parts run across the lanes, while a
// sum adds the lanes' terms one by one in index order, so it rounds as the sequential
// loop does.  One thread per cone had every division and load in one chain
// (k_nt_scaling: 166 µs for 100 cones of order 64, 17 with a warp each).
struct Lanes {
  int g, lane;  // group size, lane in the group
  unsigned mask;
  __device__ explicit Lanes(int g_) : g(g_), lane(threadIdx.x & (g_ - 1)) {
    mask = (g == 32 ? 0xffffffffu : ((1u << g) - 1)) << (threadIdx.x & 31 & ~(g - 1));
  }
  __device__ bool all(bool p) const { return __all_sync(mask, p); }
  __device__ double max(double v) const {
    for (int o = g >> 1; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(mask, v, o, g));
    return v;
  }
  // acc + the terms of the first cnt lanes, in their order.
  __device__ double fold(double acc, double term, int cnt) const {
#pragma unroll 8
    for (int k = 0; k < cnt; ++k) acc += __shfl_sync(mask, term, k, g);
    return acc;
  }
  // acc + f(i) for i = 1 … n−1, in that order.
  template <class F>
  __device__ double sum(double acc, int n, F f) const {
    for (int i0 = 1; i0 < n; i0 += g) acc = fold(acc, i0 + lane < n ? f(i0 + lane) : 0.0, min(g, n - i0));
    return acc;
  }
  // max(start, f(i)) over i = 1 … n−1.
  template <class F>
  __device__ double maximum(double start, int n, F f) const {
    for (int i = 1 + lane; i < n; i += g) start = fmax(start, f(i));
    return max(start);
  }
  template <class F>
  __device__ bool every(int n, F f) const {  // f(i) for i = 0 … n−1
    bool ok = true;
    for (int i = lane; i < n; i += g) ok = ok && f(i);
    return all(ok);
  }
};

// ------------------------------------------------------------ NT scaling --
// `_soc_tail_norm` (src/soc_lorentz_kernels.jl:21-34).
__device__ double tail_norm(const Lanes& L, const double* v, int n) {
  const double scale = L.maximum(0.0, n, [&](int i) { return fabs(v[i]); });
  if (scale == 0.0) return scale;
  const double ss = L.sum(0.0, n, [&](int i) {
    double y = v[i] / scale;
    return y * y;
  });
  return scale * sqrt(ss);
}

// `_soc_sqrt_determinant` (src/soc_lorentz_kernels.jl:42-62).
__device__ bool sqrt_determinant(const Lanes& L, const double* v, int n, double* out) {
  if (!L.every(n, [&](int i) { return isfinite(v[i]); })) return false;
  const double scale = L.maximum(fabs(v[0]), n, [&](int i) { return fabs(v[i]); });
  if (scale == 0.0) return false;
  double head = v[0];
  double tail = tail_norm(L, v, n);
  double margin = head - tail;
  if (!(margin > 0.0)) return false;
  double residual = (margin / scale) * (head / scale + tail / scale);
  if (!(residual > 0.0)) return false;
  double r = scale * sqrt(residual);
  *out = r;
  return isfinite(r) && r > 0.0;
}

// `_soc_nt_scaling!` (src/soc_lorentz_kernels.jl:72-185), g lanes per cone.
// The normalised points a = s/√det s, b = z/√det z and the midpoint raw are
// recomputed where the reference reads its temporaries (the same division
// gives the same value).  Outputs are written only after every check passed.
__global__ void k_nt_scaling(int g, int ncones, const long long* __restrict__ off,
                             const int* __restrict__ dim, const double* __restrict__ s,
                             const double* __restrict__ z, double* w, double* lam, double* eta_out,
                             double* eta2_out, int* ok_out) {
  const Lanes L(g);
  int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) / g);
  if (c >= ncones) return;
  const int n = dim[c];
  const double* sc = s + off[c];
  const double* zc = z + off[c];
  double* wc = w + off[c];
  double* lc = lam + off[c];
  if (L.lane == 0) {
    ok_out[c] = 0;
    eta_out[c] = 0.0;
    eta2_out[c] = 0.0;
  }
  double ss = 0.0, zs = 0.0;
  bool sok = sqrt_determinant(L, sc, n, &ss);
  bool zok = sqrt_determinant(L, zc, n, &zs);
  if (!(sok && zok)) return;
  double eta = sqrt(ss) / sqrt(zs);
  double eta2 = eta * eta;
  if (!(isfinite(eta2) && eta2 > 0.0)) return;
  auto A = [&](int i) { return sc[i] / ss; };
  auto B = [&](int i) { return zc[i] / zs; };
  if (!L.every(n, [&](int i) {
        double a = A(i), b = B(i);
        double raw = (i == 0) ? a + b : a - b;
        return isfinite(a) && isfinite(b) && isfinite(raw);
      }))
    return;
  const double a0 = A(0), b0 = B(0);
  const double tmax = L.maximum(0.0, n, [&](int i) { return fmax(fabs(A(i)), fabs(B(i))); });
  const double mscale = fmax(fmax(1.0, tmax), fmax(fabs(a0), fabs(b0)));
  double inv_m = 1.0 / mscale;
  double cross = L.sum((a0 * inv_m) * (b0 * inv_m), n,
                       [&](int i) { return (A(i) * inv_m) * (B(i) * inv_m); });
  double radicand = inv_m * inv_m + cross;
  if (!(isfinite(radicand) && radicand > 0.0)) return;
  double wscale = sqrt(2.0) * mscale * sqrt(radicand);
  if (!(isfinite(wscale) && wscale > 0.0)) return;
  const double nts = L.maximum(1.0, n, [&](int i) { return fabs((A(i) - B(i)) / wscale); });
  double inv_t = 1.0 / nts;
  double hacc = L.sum(inv_t * inv_t, n, [&](int i) {
    double val = ((A(i) - B(i)) / wscale) / nts;
    return val * val;
  });
  double nhead = nts * sqrt(hacc);
  if (!(isfinite(nhead) && nhead > 0.0)) return;
  double gamma = wscale / 2.0;
  double lscale = fmax(fmax(1.0, fabs(a0)), fmax(fabs(b0), fabs(gamma)));
  lscale = fmax(lscale, tmax);
  double inv_l = 1.0 / lscale;
  double aa_h = a0 * inv_l, bb_h = b0 * inv_l, gg = gamma * inv_l;
  double den = aa_h + bb_h + 2.0 * gg;
  if (!(isfinite(den) && den > 0.0)) return;
  double geo = sqrt(ss) * sqrt(zs);
  double lam_head = geo * gamma;
  if (!isfinite(lam_head)) return;
  auto lambda_i = [&](int i) {
    double aa = A(i) * inv_l, bb = B(i) * inv_l;
    double scaled = (gg + bb_h) * aa + (gg + aa_h) * bb;
    return geo * (scaled / den) * lscale;
  };
  if (!L.every(n, [&](int i) { return i == 0 || isfinite(lambda_i(i)); })) return;
  for (int i = L.lane; i < n; i += g) {
    lc[i] = i ? lambda_i(i) : lam_head;
    wc[i] = i ? (A(i) - B(i)) / wscale : nhead;
  }
  if (L.lane == 0) {
    eta_out[c] = eta;
    eta2_out[c] = eta2;
    ok_out[c] = 1;
  }
}

// ------------------------------------------------------------- NT maps ----
// `_soc_nt_apply_w!` (which = 0) / `_soc_nt_apply_winv!` (1) /
// `_soc_nt_apply_hs_inverse!` (2) (src/soc_lorentz_kernels.jl:187-255) on a cone
// vector v[0..n), by the lanes of a group.  which = 2 may add the result to `base`
// (out = base + Hs⁻¹v); W and W⁻¹ ignore it.
__device__ __forceinline__ void nt_map(const Lanes& L, int which, const double* wc, double eta, double eta2,
                                       const double* v, double* out, int n, const double* base) {
  const double head = v[0], w0 = wc[0];
  if (which == 2) {
    const double ld = L.sum(w0 * head, n, [&](int i) { return -(wc[i] * v[i]); });
    for (int i = L.lane; i < n; i += L.g) {
      double o = i ? (-2.0 * wc[i] * ld + v[i]) / eta2 : (2.0 * w0 * ld - head) / eta2;
      out[i] = base ? base[i] + o : o;
    }
    return;
  }
  const double dt = L.sum(0.0, n, [&](int i) { return wc[i] * v[i]; });
  if (which == 0) {
    double corr = head + dt / (1.0 + w0);
    for (int i = L.lane; i < n; i += L.g) out[i] = i ? eta * (v[i] + corr * wc[i]) : eta * (w0 * head + dt);
  } else {
    double corr = -head + dt / (1.0 + w0);
    for (int i = L.lane; i < n; i += L.g) out[i] = i ? (v[i] + corr * wc[i]) / eta : (w0 * head - dt) / eta;
  }
}

// The same maps (which = 0, 1) by one thread.
__device__ __forceinline__ void nt_map(int which, const double* wc, double eta, const double* v, double* out,
                                       int n) {
  const double head = v[0];
  double dt = 0.0;
  for (int i = 1; i < n; ++i) dt += wc[i] * v[i];
  if (which == 0) {
    double corr = head + dt / (1.0 + wc[0]);
    out[0] = eta * (wc[0] * head + dt);
    for (int i = 1; i < n; ++i) out[i] = eta * (v[i] + corr * wc[i]);
  } else {
    double corr = -head + dt / (1.0 + wc[0]);
    out[0] = (wc[0] * head - dt) / eta;
    for (int i = 1; i < n; ++i) out[i] = (v[i] + corr * wc[i]) / eta;
  }
}

__global__ void k_nt_apply(int g, int which, int ncones, const long long* __restrict__ off,
                           const int* __restrict__ dim, const double* __restrict__ w,
                           const double* __restrict__ eta, const double* __restrict__ eta2,
                           const double* __restrict__ v, double* __restrict__ out) {
  const Lanes L(g);
  int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) / g);
  if (c >= ncones) return;
  nt_map(L, which, w + off[c], eta[c], eta2[c], v + off[c], out + off[c], dim[c], nullptr);
}

// --------------------------------------------------------------- LP pack --
__global__ void k_lp_pack(int n_lp, const double* __restrict__ weights, const int* __restrict__ row,
                          const double* __restrict__ coef, double reg, double* D, double* Dinv,
                          double* Dis) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_lp) return;
  double c = coef[j];
  double d = weights[row[j]] * c * c + reg;
  double inv = 1.0 / d;
  D[j] = d;
  Dinv[j] = inv;
  Dis[j] = sqrt(inv);
}

// B̂[j, e] = D^{-1/2}_j · B[j, e] for the LP rows of every column: a thread keeps its
// row's factor for eight columns, whose loads are in flight together (one element a
// thread with a 64-bit division for its place: 230 µs at 20000 × 3000, now 142;
// the 960 MB take 149 at the copy rate).
constexpr int kLpCols = 8;
__global__ void k_scale_lp(int n_lp, long long n, int m, const double* __restrict__ B,
                           const double* __restrict__ Dis, double* __restrict__ Bh) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_lp) return;
  const double d = Dis[j];
  for (int c0 = blockIdx.y * kLpCols; c0 < m; c0 += gridDim.y * kLpCols) {
    const double* src = B + c0 * n + j;
    double* dst = Bh + c0 * n + j;
    double v[kLpCols];
#pragma unroll
    for (int c = 0; c < kLpCols; ++c) v[c] = c0 + c < m ? src[c * n] : 0.0;
#pragma unroll
    for (int c = 0; c < kLpCols; ++c)
      if (c0 + c < m) dst[c * n] = d * v[c];
  }
}

// B̂_k[:, e] = W_k⁻¹ B_k[:, e] for the cones of one tile (whole cones, at most kConeRows
// rows, or one larger cone) and kConeCols columns.  The rows pass through shared memory,
// so that global accesses run along the columns; a (cone, column) sum is one thread's,
// in index order.  A thread per (cone, column) walking its rows in global memory took
// 400 µs for 100 cones of order 64 and 3000 columns, this takes 98.
constexpr int kConeRows = 64, kConeCols = 32, kConeLd = kConeRows + 1;
struct ConeTile {
  int cone, ncones, row, rows;
};
__global__ void __launch_bounds__(256) k_scale_cones(const ConeTile* __restrict__ tiles, int m, long long n,
                                                     long long cone_base, const long long* __restrict__ off,
                                                     const int* __restrict__ dim, const double* __restrict__ w,
                                                     const double* __restrict__ eta,
                                                     const double* __restrict__ B, double* __restrict__ Bh) {
  __shared__ double buf[kConeCols * kConeLd], corr[kConeRows * kConeCols], ws[kConeRows], es[kConeRows];
  __shared__ int head[kConeRows];  // per row: the cone's first row, its place in the tile
  __shared__ int cone_of[kConeRows];
  const ConeTile T = tiles[blockIdx.x];
  const int tid = threadIdx.x, row = tid & (kConeRows - 1), cg = tid / kConeRows;
  const int c0 = blockIdx.y * kConeCols, cols = min(kConeCols, m - c0);
  const long long base = (long long)c0 * n + cone_base + T.row;
  const int nchunk = (T.rows + kConeRows - 1) / kConeRows;
  auto load = [&](int r0) {  // rows r0 … of the tile into buf, their w into ws
    const int r = r0 + row;
    double v[kConeCols / 4];
#pragma unroll
    for (int q = 0; q < kConeCols / 4; ++q) {
      const int c = cg + 4 * q;
      v[q] = r < T.rows && c < cols ? B[base + c * n + r] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kConeCols / 4; ++q) buf[(cg + 4 * q) * kConeLd + row] = v[q];
    if (tid < kConeRows) ws[tid] = r < T.rows ? w[T.row + r] : 0.0;
  };
  for (int q = tid; q < T.ncones; q += blockDim.x) {
    const int c = T.cone + q, first = (int)(off[c] - T.row), last = min(kConeRows, first + dim[c]);
    es[q] = eta[c];
    for (int r = first; r < last; ++r) head[r] = first, cone_of[r] = q;
  }
  load(0);
  __syncthreads();
  double hv = 0.0, dt = 0.0;  // of one larger cone: column tid
  if (nchunk == 1) {
    for (int p = tid; p < T.ncones * kConeCols; p += blockDim.x) {
      const int q = p / kConeCols, c = p % kConeCols, first = (int)(off[T.cone + q] - T.row);
      const int nq = dim[T.cone + q];
      double* v = buf + c * kConeLd + first;
      const double *wq = ws + first, h = v[0];
      double t = 0.0;
      for (int i = 1; i < nq; ++i) t += wq[i] * v[i];
      corr[p] = -h + t / (1.0 + wq[0]);
      v[0] = (wq[0] * h - t) / es[q];
    }
  } else {
    for (int k = 0; k < nchunk; ++k) {
      if (k) {
        __syncthreads();
        load(k * kConeRows);
        __syncthreads();
      }
      if (tid < kConeCols) {
        const double* v = buf + tid * kConeLd;
        if (k == 0) hv = v[0];
        const int e = min(kConeRows, T.rows - k * kConeRows);
        for (int i = k == 0; i < e; ++i) dt += ws[i] * v[i];
      }
    }
    __syncthreads();
    load(0);
    __syncthreads();
    if (tid < kConeCols) {
      corr[tid] = -hv + dt / (1.0 + ws[0]);
      buf[tid * kConeLd] = (ws[0] * hv - dt) / es[0];
    }
  }
  for (int k = 0; k < nchunk; ++k) {
    if (k) {
      __syncthreads();
      load(k * kConeRows);
    }
    __syncthreads();
    const int r = k * kConeRows + row;
    if (r >= T.rows) continue;
    const int first = nchunk == 1 ? head[row] : -k * kConeRows, q = nchunk == 1 ? cone_of[row] : 0;
    const double wr = ws[row], e = es[q];
#pragma unroll
    for (int j = 0; j < kConeCols / 4; ++j) {
      const int c = cg + 4 * j;
      const double v = buf[c * kConeLd + row];
      if (c < cols) Bh[base + c * n + r] = row == first ? v : (v + corr[q * kConeCols + c] * wr) / e;
    }
  }
}

// Q_ii += δ (Q holds the lower triangle from the SYRK); F = lower(Q).  The strict upper
// triangle of F is left to the factorization, which zeroes it.
__global__ void k_shift_copy_lower(int m, double* Q, double reg, double* F) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  for (int j0 = blockIdx.y * kLpCols; j0 <= i; j0 += gridDim.y * kLpCols) {
    double v[kLpCols];
#pragma unroll
    for (int c = 0; c < kLpCols; ++c) v[c] = j0 + c <= i ? Q[(size_t)(j0 + c) * m + i] : 0.0;
#pragma unroll
    for (int c = 0; c < kLpCols; ++c) {
      if (j0 + c > i) continue;
      const size_t e = (size_t)(j0 + c) * m + i;
      if (j0 + c == i) Q[e] = v[c] = v[c] + reg;
      F[e] = v[c];
    }
  }
}

// out = base + D⁻¹ v over all variables: LP entries by D⁻¹_j, cone k by Hs_k⁻¹
// (a thread per LP entry in the first lp_blocks blocks, then g lanes per cone).
__global__ void k_apply_dinv(int g, int lp_blocks, int n_lp, const double* __restrict__ Dinv, int ncones,
                             long long cone_base, const long long* __restrict__ off,
                             const int* __restrict__ dim, const double* __restrict__ w,
                             const double* __restrict__ eta2, const double* __restrict__ v,
                             const double* __restrict__ base, double* __restrict__ out) {
  if ((int)blockIdx.x < lp_blocks) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_lp) return;
    double o = Dinv[t] * v[t];
    out[t] = base ? base[t] + o : o;
    return;
  }
  const Lanes L(g);
  const int c = (int)(((blockIdx.x - lp_blocks) * blockDim.x + threadIdx.x) / g);
  if (c >= ncones) return;
  long long o = cone_base + off[c];
  nt_map(L, 2, w + off[c], 0.0, eta2[c], v + o, out + o, dim[c], base ? base + o : nullptr);
}

// Results of a call into pinned host memory in one launch: the four vectors one after
// the other, then the flags.  Bound by the posted writes over PCIe (0.5 MB at most); eight
// copies to pageable memory took 10 µs of the host each: a pass of the
// normal system of m = 317 (scaling, factor, solve) took 381 µs, 305 now.
struct ResultList {
  const double* src[4];
  long long n[4];
  const int* flags;
  int nflags;
};
__global__ void k_results(ResultList L, double* __restrict__ dst, int* __restrict__ dflags) {
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long step = (long long)gridDim.x * blockDim.x;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    for (long long i = t0; i < L.n[q]; i += step) dst[i] = L.src[q][i];
    dst += L.n[q];
  }
  for (long long i = t0; i < L.nflags; i += step) dflags[i] = L.flags[i];
}

}  // namespace

// ============================================================================
struct NormalHandle {
  int dev = 0;
  cudaStream_t st = nullptr;
  int sms = 148;
  std::string err;
  int n_lp = 0, ncones = 0, m = 0, n_weights = 0;
  int lanes = 4, cone_tiles = 0;  // lanes per cone, tiles of k_scale_cones
  long long n = 0, nq = 0;  // variables, cone variables
  std::vector<long long> cone_off;
  std::vector<int> cone_dim;
  DBuf<long long> d_off;
  DBuf<int> d_dim, d_row, d_ok;
  DBuf<int> d_info;  // of the factor; [1]: a wait of the triangular solve gave up
  DBuf<ConeTile> d_tiles;
  FlowFlags flow_flags;  // tile flags of the Cholesky launch
  DBuf<double> B, Bh, coef, weights, D, Dinv, Dis, w, lam, eta, eta2, sz, v, out;
  DBuf<double> Q, F, Finv_diag, partial, rhs, t, red, work, u, gemv_part;
  DBuf<double> dmin, dmax;
  // Pinned staging of a call's vectors, kHeader bytes for flags before them.  Calls with
  // more than kStageBytes copy from and to the caller's memory, as pinning megabytes costs
  // a new handle milliseconds.  Every call that uses it waits for the stream before it returns.
  static constexpr size_t kStageBytes = 1 << 20, kHeader = 64;
  PinnedBuf pin;
  size_t pin_doubles = 0;
  double* stage(long long doubles) {
    return (size_t)doubles <= pin_doubles ? reinterpret_cast<double*>(pin.p + kHeader) : nullptr;
  }
  int* pin_flags() { return reinterpret_cast<int*>(pin.p); }
  SyrkPlan plan;
  int gemv_chunks = 8;
  bool have_scaling = false, have_factor = false, have_assembled = false;
  bool standard_rows = true;  // row_for_variable = identity, g = 1, one weight per LP variable
  // Split-BF16 assembly: three BF16 planes of B̂ (m rows of pitch Kp = n
  // rounded up to 64) and the tcgen05 SYRK of the Schur path.
  long long Kp = 0;
  DBuf<unsigned char> plane_buf[3];
  SplitSyrkPlan splan;
  DBuf<float> spartial;
  DBuf<int> serr;
  // Explicit inverse of the reduced factor for the refined (mixed) solves:
  // each solve is two GEMVs over L⁻¹ instead of 2·⌈m/64⌉ dependent launches.
  DBuf<double> Linv, Ltmp;
  bool have_inverse = false;
  void make_inverse() {
    if (Linv.n < (size_t)m * m) {
      Linv.alloc((size_t)m * m);
      Linv.zero(st);
      Ltmp.alloc((size_t)m * m);
    }
    TrinvList q;
    q.count = 1;
    q.n[0] = m;
    q.L[0] = F.p;
    q.W[0] = Linv.p;
    q.tmp[0] = Ltmp.p;
    trinv(q, st);
    have_inverse = true;
  }
  // v ← Q⁻¹v = L⁻ᵀ(L⁻¹v) with the explicit inverse (work: m).
  void solve_inverse(double* v) {
    gemv_n(Linv.p, m, m, v, work.p, gemv_part.p, gemv_chunks, st);
    gemv_t(Linv.p, m, m, work.p, 1.0, nullptr, 0.0, v, st);
  }
  cudaEvent_t ev[4] = {};
  double assemble_ms = 0.0, factor_ms = 0.0;

  void create(int n_lp_, int ncones_, const int* dims, int m_, const double* hB, const int* row,
              const double* hcoef, int n_weights_, int device) {
    if (n_lp_ < 0 || ncones_ < 0 || m_ < 0 || n_weights_ < 0)
      throw std::invalid_argument("negative size");
    if (ncones_ > 0 && !dims) throw std::invalid_argument("cone_dims is NULL");
    if (n_lp_ > 0 && (!row || !hcoef || n_weights_ <= 0))
      throw std::invalid_argument("LP variables need row_for_variable, diagonal_coefficient, weights");
    dev = device;
    SDPX_CUDA(cudaSetDevice(dev));
    SDPX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SDPX_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    for (auto& e : ev) SDPX_CUDA(cudaEventCreate(&e));
    n_lp = n_lp_;
    ncones = ncones_;
    m = m_;
    n_weights = n_weights_;
    long long o = 0;
    for (int c = 0; c < ncones; ++c) {
      if (dims[c] < 1) throw std::invalid_argument("cone dimension must be >= 1");
      cone_off.push_back(o);
      cone_dim.push_back(dims[c]);
      o += dims[c];
    }
    nq = o;
    n = n_lp + nq;
    for (int j = 0; j < n_lp; ++j)
      if (row[j] < 0 || row[j] >= n_weights)
        throw std::invalid_argument("row_for_variable out of range at variable " + std::to_string(j));
    standard_rows = n_weights == n_lp;
    for (int j = 0; j < n_lp && standard_rows; ++j) standard_rows = row[j] == j && hcoef[j] == 1.0;
    if (n > 0 && m > 0 && !hB) throw std::invalid_argument("B is NULL");
    B.alloc((size_t)n * m);
    Bh.alloc((size_t)n * m);
    if (n > 0 && m > 0) h2d(B.p, hB, sizeof(double) * n * m);
    d_off.alloc(ncones);
    d_dim.alloc(ncones);
    if (ncones) {
      h2d(d_off.p, cone_off.data(), sizeof(long long) * ncones);
      h2d(d_dim.p, cone_dim.data(), sizeof(int) * ncones);
      while (lanes < 32 && (long long)lanes * ncones < nq) lanes *= 2;  // about the mean order
      std::vector<ConeTile> tiles;
      for (int c = 0; c < ncones; ++c) {
        const int q = cone_dim[c];
        if (tiles.empty() || tiles.back().rows + q > kConeRows)
          tiles.push_back({c, 1, (int)cone_off[c], q});
        else
          tiles.back().ncones++, tiles.back().rows += q;
      }
      cone_tiles = (int)tiles.size();
      d_tiles.alloc(cone_tiles);
      h2d(d_tiles.p, tiles.data(), sizeof(ConeTile) * cone_tiles);
    }
    d_row.alloc(n_lp);
    coef.alloc(n_lp);
    if (n_lp) {
      h2d(d_row.p, row, sizeof(int) * n_lp);
      h2d(coef.p, hcoef, sizeof(double) * n_lp);
    }
    weights.alloc(n_weights);
    for (auto* b : {&D, &Dinv, &Dis}) b->alloc(n_lp);
    for (auto* b : {&w, &lam, &v, &out}) b->alloc(nq);
    sz.alloc(2 * nq);
    for (auto* b : {&eta, &eta2}) b->alloc(ncones);
    d_ok.alloc(ncones);
    Q.alloc((size_t)m * m);
    F.alloc((size_t)m * m);
    Finv_diag.alloc((size_t)ceil_div(std::max(m, 1), 64) * 64 * 64);
    rhs.alloc(n + m);
    t.alloc(n);
    u.alloc(n);
    red.alloc(m);
    work.alloc(cholesky_solve_work(m));
    gemv_chunks = std::max(1, std::min(16, m / 64));
    gemv_part.alloc((size_t)gemv_chunks * std::max<long long>(n, m));
    plan = plan_syrk_f64(std::max(m, 1), std::max<long long>(n, 1), sms);
    partial.alloc(plan.partial_doubles);
    d_info.alloc(2);
    SDPX_CUDA(cudaMemsetAsync(d_info.p, 0, 2 * sizeof(int), st));
    dmin.alloc(1);
    dmax.alloc(1);
    const size_t most = std::max<size_t>({4 * (size_t)nq + 3 * (size_t)ncones, (size_t)n_weights,
                                          (size_t)(n + m)});
    pin_doubles = std::min(most, (kStageBytes - kHeader) / sizeof(double));
    pin.alloc(kHeader + pin_doubles * sizeof(double));
    sync();
  }
  ~NormalHandle() {
    if (st) {
      cudaSetDevice(dev);
      if (cudaStreamSynchronize(st) == cudaSuccess) pin.release();
      for (auto& e : ev)
        if (e) cudaEventDestroy(e);
      cudaStreamDestroy(st);
    }
  }

  void h2d(void* d, const void* h, size_t bytes) {
    if (bytes) SDPX_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st));
  }
  void d2h(void* h, const void* d, size_t bytes) {
    if (bytes) SDPX_CUDA(cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, st));
  }
  void sync() { SDPX_CUDA(cudaStreamSynchronize(st)); }

  void results(const ResultList& L, double* dst, int* flags) {
    const long long most = std::max(std::max(L.n[0], L.n[1]), std::max<long long>(L.n[2], L.nflags));
    k_results<<<std::min(32, ceil_div(most, 256)), 256, 0, st>>>(L, dst, flags);
    SDPX_LAUNCH_CHECK();
  }

  void launch_nt_scaling(const double* ds, const double* dz) {
    k_nt_scaling<<<ceil_div((long long)ncones * lanes, 128), 128, 0, st>>>(
        lanes, ncones, d_off.p, d_dim.p, ds, dz, w.p, lam.p, eta.p, eta2.p, d_ok.p);
    SDPX_LAUNCH_CHECK();
  }
  // out = base + D⁻¹v (LP diag(D⁻¹), cones Hs⁻¹) on the held scaling.
  void apply_dinv(const double* dv, const double* base, double* dout) {
    const int lp_blocks = ceil_div(n_lp, 128);
    const int grid = lp_blocks + ceil_div((long long)ncones * lanes, 128);
    if (grid == 0) return;
    k_apply_dinv<<<grid, 128, 0, st>>>(lanes, lp_blocks, n_lp, Dinv.p, ncones, n_lp, d_off.p, d_dim.p, w.p,
                                       eta2.p, dv, base, dout);
    SDPX_LAUNCH_CHECK();
  }

  int nt_scaling(const double* hs, const double* hz, int* ok, double* hw, double* hlam,
                 double* heta, double* heta2) {
    have_scaling = false;
    if (ncones == 0) return 0;
    if (!hs || !hz) throw std::invalid_argument("s and z are required");
    const size_t bytes = sizeof(double) * nq;
    std::vector<int> okv;
    const int* hok;
    if (double* h = stage(4 * nq + 3 * (long long)ncones)) {
      std::memcpy(h, hs, bytes);
      std::memcpy(h + nq, hz, bytes);
      h2d(sz.p, h, 2 * bytes);
      launch_nt_scaling(sz.p, sz.p + nq);
      const double* r = h + 2 * nq;
      int* flags = reinterpret_cast<int*>(h + 4 * nq + 2 * ncones);
      results({{w.p, lam.p, eta.p, eta2.p}, {nq, nq, ncones, ncones}, d_ok.p, ncones}, h + 2 * nq, flags);
      sync();
      if (hw) std::memcpy(hw, r, bytes);
      if (hlam) std::memcpy(hlam, r + nq, bytes);
      if (heta) std::memcpy(heta, r + 2 * nq, sizeof(double) * ncones);
      if (heta2) std::memcpy(heta2, r + 2 * nq + ncones, sizeof(double) * ncones);
      hok = flags;
    } else {
      h2d(sz.p, hs, bytes);
      h2d(sz.p + nq, hz, bytes);
      launch_nt_scaling(sz.p, sz.p + nq);
      okv.resize(ncones);
      d2h(okv.data(), d_ok.p, sizeof(int) * ncones);
      if (hw) d2h(hw, w.p, bytes);
      if (hlam) d2h(hlam, lam.p, bytes);
      if (heta) d2h(heta, eta.p, sizeof(double) * ncones);
      if (heta2) d2h(heta2, eta2.p, sizeof(double) * ncones);
      sync();
      hok = okv.data();
    }
    int bad = 0;
    for (int c = 0; c < ncones; ++c) {
      if (ok) ok[c] = hok[c];
      bad += hok[c] == 0;
    }
    have_scaling = bad == 0;
    have_factor = false;
    return bad ? 1 : 0;
  }

  void require_scaling() {
    if (ncones > 0 && !have_scaling)
      throw std::logic_error("no valid NT scaling held: call nt_scaling with interior points first");
  }

  void nt_apply(int which, const double* hv, double* hout) {
    if (which < 0 || which > 2) throw std::invalid_argument("which must be 0 (W), 1 (W^-1) or 2 (Hs^-1)");
    require_scaling();
    if (ncones == 0) return;
    h2d(v.p, hv, sizeof(double) * nq);
    k_nt_apply<<<ceil_div((long long)ncones * lanes, 128), 128, 0, st>>>(
        lanes, which, ncones, d_off.p, d_dim.p, w.p, eta.p, eta2.p, v.p, out.p);
    SDPX_LAUNCH_CHECK();
    d2h(hout, out.p, sizeof(double) * nq);
    sync();
  }

  void pack(const double* hweights, double reg) {
    if (n_lp == 0) return;
    if (!hweights) throw std::invalid_argument("weights is NULL");
    const size_t bytes = sizeof(double) * n_weights;
    if (double* h = stage(n_weights)) hweights = static_cast<const double*>(std::memcpy(h, hweights, bytes));
    h2d(weights.p, hweights, bytes);
    k_lp_pack<<<ceil_div(n_lp, 256), 256, 0, st>>>(n_lp, weights.p, d_row.p, coef.p, reg, D.p,
                                                    Dinv.p, Dis.p);
    SDPX_LAUNCH_CHECK();
  }

  // B̂ rows of the cones (independent of δ) — once per scaling.
  void scale_cones() {
    if (ncones == 0 || m == 0) return;
    // Column tiles in slices, for the grid's y extent.
    for (int c0 = 0; c0 < m; c0 += 65535 * kConeCols) {
      const int cols = std::min(m - c0, 65535 * kConeCols);
      k_scale_cones<<<dim3(cone_tiles, ceil_div(cols, kConeCols)), 256, 0, st>>>(
          d_tiles.p, cols, n, n_lp, d_off.p, d_dim.p, w.p, eta.p, B.p + (size_t)c0 * n, Bh.p + (size_t)c0 * n);
      SDPX_LAUNCH_CHECK();
    }
  }

  // Q = B̂ᵀB̂ from three BF16 planes of B̂ on the tcgen05 split SYRK (FP32
  // tiles summed in FP64; ≈ 1e-6 relative), +δ and the lower copy into F.
  void assemble_split(double reg) {
    if (m == 0) return;
    scale_lp_rows();
    if (Kp == 0) {
      Kp = (std::max<long long>(n, 1) + 63) / 64 * 64;
      for (auto& b : plane_buf) b.alloc(sizeof(__nv_bfloat16) * (size_t)m * Kp);
      splan = plan_split_syrk(m, Kp, sms);
      spartial.alloc(splan.partial_floats);
      serr.alloc(1);
    }
    __nv_bfloat16* pl[3];
    for (int i = 0; i < 3; ++i) pl[i] = reinterpret_cast<__nv_bfloat16*>(plane_buf[i].p);
    split_rows_f64(Bh.p, n, m, n, Kp, pl, st);
    SDPX_CUDA(cudaMemsetAsync(serr.p, 0, sizeof(int), st));
    Plane2D P{{pl[0], pl[1], pl[2]}, m, Kp};
    split_syrk(P, m, (int)Kp, splan, spartial.p, Q.p, serr.p, st);
    int e = 0;
    d2h(&e, serr.p, sizeof(int));
    sync();
    if (e) throw CudaError("split normal-matrix SYRK: a bounded wait gave up");
    shift_copy(reg);
  }

  // +δ on the diagonal of Q, copy of lower(Q) into F.
  void shift_copy(double reg) {
    const dim3 grid(ceil_div(m, 256), std::min(65535, ceil_div(m, kLpCols)));
    k_shift_copy_lower<<<grid, 256, 0, st>>>(m, Q.p, reg, F.p);
    SDPX_LAUNCH_CHECK();
    have_assembled = true;
  }

  // B̂ = D^{-1/2}B on the LP rows (the cone rows come from scale_cones).
  void scale_lp_rows() {
    if (n_lp > 0 && m > 0) {
      const dim3 grid(ceil_div(n_lp, 256), std::min(65535, ceil_div(m, kLpCols)));
      k_scale_lp<<<grid, 256, 0, st>>>(n_lp, n, m, B.p, Dis.p, Bh.p);
      SDPX_LAUNCH_CHECK();
    }
  }

  // LP rows of B̂, SYRK, +δ on the diagonal, copy of lower(Q) into F.
  void assemble_lp_and_syrk(double reg) {
    if (m == 0) return;
    scale_lp_rows();
    if (n > 0) {
      Opnd P;
      P.base = Bh.p;
      P.kstride = 1;
      P.inner = 1 << 30;
      P.inner_stride = n;
      P.outer_stride = 0;
      P.mn_extent = m;
      P.k_extent = (int)n;
      syrk_lower_f64(P, plan, partial.p, Q.p, m, m, 0.0, st);
    } else {
      SDPX_CUDA(cudaMemsetAsync(Q.p, 0, sizeof(double) * (size_t)m * m, st));
    }
    shift_copy(reg);
  }

  void assemble(const double* hweights, double reg) {
    require_scaling();
    have_factor = false;
    SDPX_CUDA(cudaEventRecord(ev[0], st));
    pack(hweights, reg);
    scale_cones();
    assemble_lp_and_syrk(reg);
    SDPX_CUDA(cudaEventRecord(ev[1], st));
    sync();
    float ms = 0.f;
    SDPX_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
    assemble_ms = ms;
  }

  // Returns 0 on success, 1 when every attempt failed.
  int factorize(const double* hweights, double reg, int max_attempts, int* attempts,
                double* reg_used) {
    if (max_attempts < 1) throw std::invalid_argument("max_attempts must be >= 1");
    require_scaling();
    have_factor = false;
    double r = reg;
    int info = 1;
    int att = 0;
    float asm_ms = 0.f, fac_ms = 0.f;
    for (att = 1; att <= max_attempts; ++att) {
      SDPX_CUDA(cudaEventRecord(ev[0], st));
      pack(hweights, r);
      if (att == 1) scale_cones();
      assemble_lp_and_syrk(r);
      SDPX_CUDA(cudaEventRecord(ev[1], st));
      if (m == 0) {
        info = 0;
        break;
      }
      factor_F();
      SDPX_CUDA(cudaEventRecord(ev[2], st));
      factor_diag_inverses(F.p, m, m, Finv_diag.p, st);  // one wait for both; unused if F failed
      info = read_info();
      float a = 0.f, f = 0.f;
      SDPX_CUDA(cudaEventElapsedTime(&a, ev[0], ev[1]));
      SDPX_CUDA(cudaEventElapsedTime(&f, ev[1], ev[2]));
      asm_ms += a;
      fac_ms += f;
      if (info == 0 || att == max_attempts) break;
      r *= 10.0;
    }
    if (attempts) *attempts = att;
    if (reg_used) *reg_used = r;
    assemble_ms = asm_ms;
    factor_ms = fac_ms;
    if (info != 0) return 1;
    if (m == 0) sync();
    have_factor = true;
    return 0;
  }

  // Cholesky of the reduced matrix F in place.
  void factor_F() {
    const MatDesc<double> md{F.p, m, m};
    potrf_flow(&md, nullptr, 1, m, d_info.p, dmin.p, dmax.p, flow_flags, sms, st);
  }

  // One assembly + Cholesky attempt with LP weights already on the device
  // (one weight per LP variable): 0 on success, 1 when the factor failed.
  int factorize_dev(const double* dweights, double reg, bool split = false) {
    require_scaling();
    have_factor = false;
    have_inverse = false;
    if (n_lp) {
      k_lp_pack<<<ceil_div(n_lp, 256), 256, 0, st>>>(n_lp, dweights, d_row.p, coef.p, reg, D.p,
                                                      Dinv.p, Dis.p);
      SDPX_LAUNCH_CHECK();
    }
    scale_cones();
    if (split) assemble_split(reg);
    else assemble_lp_and_syrk(reg);
    if (m == 0) {
      have_factor = true;
      return 0;
    }
    factor_F();
    if (read_info() != 0) return 1;
    factor_diag_inverses(F.p, m, m, Finv_diag.p, st);
    if (split) make_inverse();
    have_factor = true;
    return 0;
  }

  void get_matrix(int which, double* hout) {
    if (which == 0) {
      if (!have_assembled) throw std::logic_error("no assembled matrix");
      if (m > 0) mirror_lower(m, Q.p, st);
      d2h(hout, Q.p, sizeof(double) * (size_t)m * m);
    } else {
      if (!have_factor) throw std::logic_error("no successful factor held");
      d2h(hout, F.p, sizeof(double) * (size_t)m * m);
    }
    sync();
  }

  // Device-resident solve on rhs (n + m) already in `rhs`.
  void solve_device() {
    apply_dinv(rhs.p, nullptr, t.p);  // t = D⁻¹ rx
    if (m == 0) {
      if (n > 0) SDPX_CUDA(cudaMemcpyAsync(rhs.p, t.p, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
      return;
    }
    double* dy = rhs.p + n;
    // dy ← ry − Bᵀt, then Q⁻¹
    if (n > 0) gemv_t(B.p, n, m, t.p, -1.0, dy, 1.0, dy, st);
    cholesky_solve(F.p, m, m, Finv_diag.p, dy, work.p, d_info.p + 1, sms, st);
    if (n == 0) return;
    // dx = t + D⁻¹(B dy)
    gemv_n(B.p, n, m, dy, u.p, gemv_part.p, gemv_chunks, st);
    apply_dinv(u.p, t.p, rhs.p);
  }

  // Status of the factor and of the solves before it, read in one copy.
  int read_info() {
    int* info = pin_flags();
    d2h(info, d_info.p, 2 * sizeof(int));
    sync();
    check_solve(info[1]);
    if (info[0] < 0) throw CudaError("normal-matrix Cholesky: a wait for a tile gave up");
    return info[0];
  }
  void check_solve(int err) {
    if (!err) return;
    SDPX_CUDA(cudaMemsetAsync(d_info.p + 1, 0, sizeof(int), st));
    throw CudaError("normal-matrix triangular solve: a wait for a block gave up");
  }

  int solve(double* hrhs) {
    if (!have_factor) return 1;
    const size_t bytes = sizeof(double) * (n + m);
    double* h = stage(n + m);
    if (h) std::memcpy(h, hrhs, bytes);
    h2d(rhs.p, h ? h : hrhs, bytes);
    solve_device();
    int err = 0;
    if (h) {
      results({{rhs.p}, {n + m}, d_info.p + 1, 1}, h, pin_flags());
      sync();
      std::memcpy(hrhs, h, bytes);
      err = *pin_flags();
    } else {
      d2h(&err, d_info.p + 1, sizeof(int));
      d2h(hrhs, rhs.p, bytes);
      sync();
    }
    check_solve(err);
    return 0;
  }
};

}  // namespace sdpx

#include "cone_ipm.inc"

// ============================================================================
//                                   C ABI
// ============================================================================
struct sdpx_b200_normal {
  sdpx::NormalHandle h;
};

static thread_local std::string g_normal_create_error;

#define NGUARD(hh, body)                      \
  do {                                        \
    if (!(hh)) return -1;                     \
    try {                                     \
      SDPX_CUDA(cudaSetDevice((hh)->h.dev));  \
      body;                                   \
      return 0;                               \
    } catch (const std::exception& ex) {      \
      (hh)->h.err = ex.what();                \
      return -2;                              \
    } catch (...) {                           \
      (hh)->h.err = "unknown error";          \
      return -3;                              \
    }                                         \
  } while (0)

extern "C" {

int sdpx_b200_normal_create(int32_t n_lp, int32_t n_cones, const int32_t* cone_dims, int32_t m_eq,
                            const double* B, const int32_t* row_for_variable,
                            const double* diagonal_coefficient, int32_t n_weights, int device,
                            sdpx_b200_normal** out) {
  if (!out) return -1;
  *out = nullptr;
  auto* hh = new (std::nothrow) sdpx_b200_normal();
  if (!hh) return -4;
  try {
    hh->h.create(n_lp, n_cones, cone_dims, m_eq, B, row_for_variable, diagonal_coefficient,
                 n_weights, device);
  } catch (const std::exception& ex) {
    g_normal_create_error = ex.what();
    delete hh;
    return -2;
  }
  *out = hh;
  return 0;
}
void sdpx_b200_normal_destroy(sdpx_b200_normal* h) { delete h; }
const char* sdpx_b200_normal_last_error(const sdpx_b200_normal* h) {
  return h ? h->h.err.c_str() : "null handle";
}
const char* sdpx_b200_normal_create_error(void) { return g_normal_create_error.c_str(); }

int sdpx_b200_normal_nt_scaling(sdpx_b200_normal* h, const double* s, const double* z, int32_t* ok,
                                double* w, double* lambda, double* eta, double* eta_squared) {
  NGUARD(h, return h->h.nt_scaling(s, z, ok, w, lambda, eta, eta_squared));
}
int sdpx_b200_normal_nt_apply(sdpx_b200_normal* h, int32_t which, const double* v, double* out) {
  NGUARD(h, {
    h->h.nt_apply(which, v, out);
    return 0;
  });
}
int sdpx_b200_normal_pack(sdpx_b200_normal* h, const double* weights, double regularization,
                          double* D, double* inverse_diagonal, double* inverse_sqrt) {
  NGUARD(h, {
    auto& H = h->h;
    H.pack(weights, regularization);
    if (D) H.d2h(D, H.D.p, sizeof(double) * H.n_lp);
    if (inverse_diagonal) H.d2h(inverse_diagonal, H.Dinv.p, sizeof(double) * H.n_lp);
    if (inverse_sqrt) H.d2h(inverse_sqrt, H.Dis.p, sizeof(double) * H.n_lp);
    H.sync();
    return 0;
  });
}
int sdpx_b200_normal_assemble(sdpx_b200_normal* h, const double* weights, double regularization) {
  NGUARD(h, {
    h->h.assemble(weights, regularization);
    return 0;
  });
}
int sdpx_b200_normal_factorize(sdpx_b200_normal* h, const double* weights, double regularization,
                               int32_t max_attempts, int32_t* attempts,
                               double* regularization_used) {
  NGUARD(h, {
    int att = 0;
    int rc = h->h.factorize(weights, regularization, max_attempts, &att, regularization_used);
    if (attempts) *attempts = att;
    if (rc) h->h.err = "reduced normal matrix not positive definite after regularization retries";
    return rc;
  });
}
int sdpx_b200_normal_get_matrix(sdpx_b200_normal* h, int32_t which, double* out) {
  NGUARD(h, {
    if (!out) throw std::invalid_argument("out is NULL");
    h->h.get_matrix(which, out);
    return 0;
  });
}
int sdpx_b200_normal_solve(sdpx_b200_normal* h, double* rhs) {
  NGUARD(h, {
    if (!rhs) throw std::invalid_argument("rhs is NULL");
    int rc = h->h.solve(rhs);
    if (rc) h->h.err = "no successful factor held (factorize failed or was not called)";
    return rc;
  });
}
int sdpx_b200_normal_optimize(sdpx_b200_normal* h, const double* b, const double* c,
                              const sdpx_b200_solve_options* opts, sdpx_b200_solve_result* result,
                              double* x, double* y, double* z) {
  if (!h) return -1;
  try {
    SDPX_CUDA(cudaSetDevice(h->h.dev));
    if (!opts || !c || (h->h.m > 0 && !b)) throw std::invalid_argument("NULL b, c or options");
    if (!h->h.standard_rows)
      throw std::invalid_argument("the LP part must be standard form (identity rows, g = 1)");
    sdpx::ConeIPM ipm(h->h);
    ipm.run(b, c, *opts, result, x, y, z);
    return 0;
  } catch (const std::exception& ex) {
    h->h.err = ex.what();
    return -2;
  }
}
int sdpx_b200_normal_times(sdpx_b200_normal* h, double* assemble_ms, double* factor_ms) {
  NGUARD(h, {
    if (assemble_ms) *assemble_ms = h->h.assemble_ms;
    if (factor_ms) *factor_ms = h->h.factor_ms;
    return 0;
  });
}
int sdpx_b200_normal_get_stream(sdpx_b200_normal* h, void** stream) {
  NGUARD(h, {
    if (!stream) throw std::invalid_argument("stream is NULL");
    *stream = (void*)h->h.st;
    return 0;
  });
}

}  // extern "C"

// Device side of the batched small-SDP engine (batch.cu): one CTA per
// instance per phase, every instance one PSD block of order k ≤ 64 with m ≤ 256
// constraints.  Instance matrices live in HBM at per-instance offsets; the
// k×k work of a phase runs in shared memory.  The arithmetic of each phase is
// the single-instance path's (the same Newton-step stages of src/step.jl and
// src/kernels/threaded.jl restated for one block): residuals and block factors,
// the Schur panel P̂_j = L_X⁻¹A_jL_Y and S = P̂P̂ᵀ, the Schur Cholesky with
// the reference's regularisation retries, the right-hand sides, the direction
// blocks, the fraction-to-boundary bisection, refinement residuals, the
// backtracking line search with its Cholesky margin and the update.  Step-length
// trials run eight at a time, one warp each, in the bisection and in long searches of
// orders up to 32, else one after the other by the whole CTA.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"
#include "lambda_bound.cuh"
#include "tile64.cuh"

namespace sdpx {
namespace batch {

constexpr int kMaxK = 64;
constexpr int kMaxM = 256;
constexpr int kThreads = 256;

// Per-instance layout (element offsets into the pooled arrays).
struct Inst {
  int k, m;
  long long kk_off;   // k² arrays: X, Y, C, P, R, LX, LY, W, dX, dY, Z, Xb, Yb
  long long m_off;    // m arrays: c, x, dx, d, r, rho, xb, dxb
  long long mm_off;   // m² arrays: S, LS
  long long a_off;    // m·k² arrays: A (rows vec(A_j)), the Schur panel P̂
};

struct Pool {
  const Inst* inst;
  const double* A;
  double* Ph;
  const double* C;
  const double* c;
  double *X, *Y, *P, *R, *LX, *LY, *W, *dX, *dY, *Z, *Xb, *Yb;
  double *x, *dx, *d, *r, *rho, *xb, *dxb;
  double *S, *LS;
  long long kq;  // stride of one k×k matrix slot in shared memory (a padded tile64 tile of order kmax)
  long long kp;  // stride of one packed lower-triangle slot (kmax(kmax+1)/2)
  // Float64x2 mode: low halves of the double-double arrays (hi halves are the
  // FP64 arrays above), X⁻¹ in double-double and the low half of the panel.
  double *Pl, *Rl, *Zl, *dl, *rl, *dxl, *dxbl, *rhol, *Sl, *LSl, *Xih, *Xil, *Gl;
};

// |v| with NaN read as +inf, so a poisoned value never passes a max-norm test.
__device__ __forceinline__ double abs_nan_inf(double v) {
  const double a = fabs(v);
  return (a == a) ? a : 1.0 / 0.0;
}

// ------------------------------------------------------------ reductions --
__device__ inline double cta_sum(double v, double* red) { return block_sum(v, red); }
__device__ inline double cta_max(double v, double* red) { return block_max(v, red); }

// ------------------------------------------------ passes over the constraints
// One CTA reads its instance's 𝒜 (up to 6.5 MB) in every phase, so what counts is
// how many loads each thread has in flight: with one at a time the 512-instance
// residual phase took 1.5 ms, where its bytes take 0.09 ms.  Both passes issue
// 16 loads a thread before their first use; sums keep the order j = 0, 1, … .

// f(e, Σ_j x[j]·A[j·kk + e]) for the elements e of this thread (x in shared memory).
template <class F>
__device__ __forceinline__ void cta_amul(const double* A, const double* x, int m, int kk, F f) {
  constexpr int EV = 4, JU = 4;
  const int nt = blockDim.x;
  for (int e0 = threadIdx.x; e0 < kk; e0 += EV * nt) {
    double s[EV] = {};
    const double* a = A + e0;
    int j = 0;
    for (; j + JU <= m; j += JU, a += (long long)JU * kk) {
      double v[JU][EV];
#pragma unroll
      for (int u = 0; u < JU; ++u)
#pragma unroll
        for (int q = 0; q < EV; ++q) v[u][q] = e0 + q * nt < kk ? a[u * kk + q * nt] : 0.0;
#pragma unroll
      for (int u = 0; u < JU; ++u)
#pragma unroll
        for (int q = 0; q < EV; ++q) s[q] += x[j + u] * v[u][q];
    }
    for (; j < m; ++j, a += kk)
#pragma unroll
      for (int q = 0; q < EV; ++q)
        if (e0 + q * nt < kk) s[q] += x[j] * a[q * nt];
#pragma unroll
    for (int q = 0; q < EV; ++q)
      if (e0 + q * nt < kk) f(e0 + q * nt, s[q]);
  }
}

// f(j, ⟨A_j, y⟩) for every j, four constraints a warp at a time (y's elements are read
// once for the four); f runs in all lanes.
template <class F>
__device__ __forceinline__ void cta_atmul(const double* A, const double* y, int m, int kk, F f) {
  constexpr int JW = 4, U = 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int j0 = warp * JW; j0 < m; j0 += nw * JW) {
    const double* a[JW];
#pragma unroll
    for (int w = 0; w < JW; ++w) a[w] = A + (long long)min(j0 + w, m - 1) * kk;
    double s[JW] = {};
    for (int e0 = lane; e0 < kk; e0 += 32 * U) {
      double v[U][JW], yv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool in = e0 + 32 * u < kk;
        yv[u] = in ? y[e0 + 32 * u] : 0.0;
#pragma unroll
        for (int w = 0; w < JW; ++w) v[u][w] = in ? a[w][e0 + 32 * u] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (e0 + 32 * u < kk)
#pragma unroll
          for (int w = 0; w < JW; ++w) s[w] += v[u][w] * yv[u];
    }
#pragma unroll
    for (int w = 0; w < JW; ++w) {
      const double t = warp_sum(s[w]);
      if (j0 + w < m) f(j0 + w, t);
    }
  }
}

// The vector x (m) in shared memory (ends with a CTA barrier).
__device__ __forceinline__ void cta_load_vec(double* xs, const double* x, int m) {
  for (int i = threadIdx.x; i < m; i += blockDim.x) xs[i] = x[i];
  __syncthreads();
}

// ------------------------------------------------------ small factorisations
// In-place lower Cholesky of the k×k column-major M (shared memory), the
// unblocked right-looking algorithm (LAPACK potf2's operation order per column).
// Returns false at the first pivot that is not > 0 (or NaN); the upper
// triangle is left as it was.  Writes min/max |L_jj| to *dmin/*dmax on success.
__device__ bool cta_chol(double* M, int k, double* sflag, double* dmin, double* dmax) {
  for (int j = 0; j < k; ++j) {
    if (threadIdx.x == 0) {
      const double d = M[j + j * k];
      sflag[0] = d;
      sflag[1] = (d > 0.0) ? sqrt(d) : 0.0;
    }
    __syncthreads();
    const double piv = sflag[0];
    if (!(piv > 0.0)) return false;
    const double ljj = sflag[1];
    const double inv = 1.0 / ljj;
    for (int i = j + 1 + threadIdx.x; i < k; i += blockDim.x) M[i + j * k] *= inv;
    if (threadIdx.x == 0) M[j + j * k] = ljj;
    __syncthreads();
    const int rem = k - j - 1;
    for (int e = threadIdx.x; e < rem * rem; e += blockDim.x) {
      const int ii = j + 1 + e % rem, ll = j + 1 + e / rem;
      if (ii >= ll) M[ii + ll * k] -= M[ii + j * k] * M[ll + j * k];
    }
    __syncthreads();
  }
  if (dmin) {
    if (threadIdx.x == 0) {
      double mn = fabs(M[0]), mx = mn;
      for (int j = 1; j < k; ++j) {
        mn = fmin(mn, fabs(M[j + j * k]));
        mx = fmax(mx, fabs(M[j + j * k]));
      }
      sflag[0] = mn;
      sflag[1] = mx;
    }
    __syncthreads();
    *dmin = sflag[0];
    *dmax = sflag[1];
    __syncthreads();
  }
  return true;
}

// ------------------------------------------- k×k matrices in shared tiles
// The phases keep a k×k matrix (k ≤ 64) as a tile64 tile.
using tile64::FLD;
using tile64::cta_load_tile;
using tile64::cta_tile_gemm;
using tile64::cta_tile_cholsolve;
using tile64::kFull;
using tile64::kLower;
using tile64::kUpper;

// f(r, c, S(r, c)) over the k×k elements, lanes along the columns.
template <class F>
__device__ __forceinline__ void cta_each(const double* S, int k, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = warp; c < k; c += kThreads / 32)
    for (int r = lane; r < k; r += 32) f(r, c, S[c * FLD + r]);
}

// Lower Cholesky of the tile M in place (inv: reciprocal pivots).  False at a pivot
// that is not > 0 (or NaN).  min/max |L_jj| to *dmin/*dmax.  Ends with a CTA barrier.
__device__ __forceinline__ bool cta_tile_chol(double* M, int k, double* inv, int* sfail, double* dmin,
                                              double* dmax, double* red) {
  if (threadIdx.x == 0) *sfail = tile64::kNoFail;
  __syncthreads();
  tile64::factor_tile(M, inv, (k + 7) / 8, sfail);
  __syncthreads();
  if (*sfail != tile64::kNoFail) return false;
  const double v = (int)threadIdx.x < k ? M[threadIdx.x * FLD + threadIdx.x] : 0.0;
  *dmax = cta_max(v, red);
  *dmin = -cta_max((int)threadIdx.x < k ? -v : -INFINITY, red);
  return true;
}

// X ← L⁻ᵀ for the factor in D (inv: reciprocal pivots).  Ends with a CTA barrier.
__device__ __forceinline__ void cta_tile_inverse_t(double* X, const double* D, const double* inv, int nb) {
  for (int e = threadIdx.x; e < 64 * 8 * nb; e += kThreads) {
    const int r = e & 63, c = e >> 6;
    X[c * FLD + r] = r == c ? 1.0 : 0.0;
  }
  __syncthreads();
  if ((int)(threadIdx.x >> 5) < nb) tile64::solve_strip(X, D, inv, nb);
  __syncthreads();
}

// ------------------------------------------ concurrent trials, one per warp
// The step-length phases test several step lengths of one instance at once:
// the CTA stages the lower triangles of X and dX in shared memory (packed,
// column-major: column j starts at pk_off(j, k)), and each warp factors its own
// trial matrix M = X + t·dX in its own packed slot with warp barriers only.
// Per element the operations and their order are those of cta_chol (pivot,
// scale by 1/L_jj, rank-one update column by column), so a trial's outcome is
// the same.
constexpr int kTrialWarps = kThreads / 32;

__device__ __forceinline__ int pk_off(int j, int k) { return j * k - (j * (j - 1)) / 2; }

// Packed lower triangles of the k×k column-major X and dX (global) into Xp,
// dXp (shared); called by the whole CTA.
__device__ void cta_load_packed(const double* X, const double* dX, int k, double* Xp,
                                double* dXp) {
  __syncthreads();  // the previous side's trials are done with Xp, dXp
  for (int e = threadIdx.x; e < k * k; e += blockDim.x) {
    const int i = e % k, j = e / k;
    if (i >= j) {
      const int p = pk_off(j, k) + i - j;
      Xp[p] = X[e];
      dXp[p] = dX[e];
    }
  }
  __syncthreads();
}

// Next packed position 32 further down the trailing triangle: row i of
// column c, columns holding rows c..k-1.
__device__ __forceinline__ void pk_advance(int& c, int& i, int k) {
  i += 32;
  while (i >= k && c < k - 1) {
    i = i - k + c + 1;
    ++c;
  }
}

// Is Xp + t·dXp positive definite (and, for ratio > 0, min|L_jj| > ratio·max|L_jj|)?
// Called by all 32 lanes of a warp.
__device__ bool warp_trial(const double* __restrict__ Xp, const double* __restrict__ dXp,
                           double t, int k, double ratio, double* __restrict__ slot) {
  const int lane = threadIdx.x & 31;
  const int n = k * (k + 1) / 2;
#pragma unroll 4
  for (int p = lane; p < n; p += 32) slot[p] = Xp[p] + t * dXp[p];
  __syncwarp();
  double mn = 0.0, mx = 0.0;
  for (int j = 0; j < k; ++j) {
    const int oj = pk_off(j, k) - j;  // slot[oj + i] = M(i, j)
    const double d = slot[oj + j];
    if (!(d > 0.0)) return false;  // every lane read the same pivot
    const double ljj = sqrt(d);
    const double inv = 1.0 / ljj;
    mn = j == 0 ? ljj : fmin(mn, ljj);
    mx = j == 0 ? ljj : fmax(mx, ljj);
    __syncwarp();  // the pivot is read before lane 0 overwrites it
    for (int i = j + 1 + lane; i < k; i += 32) slot[oj + i] *= inv;
    if (lane == 0) slot[oj + j] = ljj;
    __syncwarp();
    // M(i, c) −= L(i, j)·L(c, j) over the trailing triangle c ≥ j+1, i ≥ c:
    // lanes walk its packed positions 32 apart, four independent updates in
    // flight per lane (their targets are distinct and column j is read only).
    const int r = k - j - 1;
    const int T = r * (r + 1) / 2;
    int c = j + 1, i = j + 1 + lane;
    while (i >= k && c < k - 1) {
      i = i - k + c + 1;
      ++c;
    }
    for (int q = lane; q < T; q += 128) {
      int cc[4], ii[4];
      cc[0] = c;
      ii[0] = i;
#pragma unroll
      for (int u = 1; u < 4; ++u) {
        pk_advance(c, i, k);
        cc[u] = c;
        ii[u] = i;
      }
      pk_advance(c, i, k);
      double tv[4], a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q + 32 * u < T) {
          tv[u] = slot[pk_off(cc[u], k) - cc[u] + ii[u]];
          a[u] = slot[oj + ii[u]];
          b[u] = slot[oj + cc[u]];
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q + 32 * u < T) slot[pk_off(cc[u], k) - cc[u] + ii[u]] = tv[u] - a[u] * b[u];
    }
    __syncwarp();
  }
  if (!(ratio > 0.0)) return true;
  return isfinite(mn) && isfinite(mx) && mx > 0.0 && mn > ratio * mx;
}

// `fraction_to_boundary_bound!` (src/kernels/generic.jl:350-422) with the
// bisection evaluated as a tree: each round tests the 7 midpoints of the next
// three bisection steps at once (warps 0..6; warp 7 tests the full step in
// the first round) and walks the tree, so the result is the sequential
// bisection's: 1 if X + dX is positive definite, else the lower end after at
// most 64 steps, stopping once [lo, hi] holds no double strictly inside.
// Called by the whole CTA (kThreads threads); sm: 2 + kTrialWarps packed
// slots of stride kp (X, dX, the trials); flags: kTrialWarps ints in shared
// memory.
__device__ double cta_ftb_tree(const double* X, const double* dX, int k, double* sm,
                               long long kp, int* flags) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* Xp = sm;
  double* dXp = sm + kp;
  double* slot = sm + (2 + w) * kp;
  cta_load_packed(X, dX, k, Xp, dXp);
  double lo = 0.0, hi = 1.0;
  int done = 0;
  bool first = true;
  while (true) {
    const int depth = min(3, 64 - done);
    const int npts = (1 << depth) - 1;
    double los[7], his[7], pts[7];
    los[0] = lo;
    his[0] = hi;
#pragma unroll
    for (int n = 0; n < 7; ++n) {
      if (n >= npts) break;
      pts[n] = (los[n] + his[n]) / 2.0;
      const int l2 = 2 * n + 1, r2 = 2 * n + 2;
      if (l2 < npts) los[l2] = los[n], his[l2] = pts[n];
      if (r2 < npts) los[r2] = pts[n], his[r2] = his[n];
    }
    if (w < npts) {
      const bool ok = warp_trial(Xp, dXp, pts[w], k, 0.0, slot);
      if (lane == 0) flags[w] = ok ? 1 : 0;
    } else if (first && w == kTrialWarps - 1) {
      const bool ok = warp_trial(Xp, dXp, 1.0, k, 0.0, slot);
      if (lane == 0) flags[w] = ok ? 1 : 0;
    }
    __syncthreads();
    int f[kTrialWarps];
#pragma unroll
    for (int n = 0; n < kTrialWarps; ++n) f[n] = flags[n];
    __syncthreads();  // every thread has its copy before the next round writes
    if (first) {
      first = false;
      if (f[kTrialWarps - 1]) return 1.0;
    }
    int node = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (node >= npts) break;
      if (f[node]) {
        lo = pts[node];
        node = 2 * node + 2;
      } else {
        hi = pts[node];
        node = 2 * node + 1;
      }
      ++done;
    }
    const double mid = (lo + hi) / 2.0;
    if (done >= 64 || mid == hi || (mid == lo && lo > 0.0)) return lo;
  }
}

// The same test for orders up to 32, without the updates of the whole triangle: lane r
// forms row r's entry of a column from the finished columns, one product after the other
// (per element the operations of warp_trial in their order).  L: a packed slot.
constexpr int kSmallTrialOrder = 32;
__device__ bool warp_trial_rows(const double* __restrict__ Xp, const double* __restrict__ dXp, double t, int k,
                                double ratio, double* __restrict__ L) {
  const int lane = threadIdx.x & 31;
  double mn = INFINITY, mx = 0.0;
  int oc = 0;  // L(i, c) at oc + i
  for (int c = 0; c < k; ++c) {
    const int r = max(min(lane, k - 1), c);
    double a = Xp[oc + r] + t * dXp[oc + r];
    int o = 0, j = 0;
    for (; j + 4 <= c; j += 4) {
      double u[4], v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        u[q] = L[o + r];
        v[q] = L[o + c];
        o += k - 1 - (j + q);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) a -= u[q] * v[q];
    }
    for (; j < c; ++j) {
      a -= L[o + r] * L[o + c];
      o += k - 1 - j;
    }
    const double d = __shfl_sync(0xffffffffu, a, c);
    if (!(d > 0.0)) return false;
    double l, inv;
    if (d > 0x1p-830 && d < 0x1p830) {
      tile64::sqrt_rcp(d, l, inv);
    } else {
      l = sqrt(d);
      inv = 1.0 / l;
    }
    mn = fmin(mn, l);
    mx = fmax(mx, l);
    if (lane >= c && lane < k) L[oc + lane] = lane == c ? l : a * inv;
    __syncwarp();
    oc += k - 1 - c;
  }
  if (!(ratio > 0.0)) return true;
  return isfinite(mn) && isfinite(mx) && mx > 0.0 && mn > ratio * mx;
}

// Backtracking (src/kernels/threaded.jl:1751-1818): the first t of 1, γ, γ², …
// whose trial X + t·dX passes (Cholesky and, for ratio > 0, the diagonal-ratio
// margin), or the first t below min_step.  γ ∈ (0, 1) reaches min_step > 0 long before
// the round guard, which bounds the loop for any other input.
//
// Trials one after the other, each by the whole CTA in one tile M, seq of them at most;
// true when one ended the search, else *t is the next candidate.  ROWS ≥ k: 32 or 64.
template <int ROWS>
__device__ __forceinline__ bool cta_trials(const double* X, const double* dX, int k, double gamma, double min_step,
                                           double ratio, int seq, double* M, double* inv, int* sfail, double* red,
                                           double* t) {
  constexpr int STEP = kThreads / ROWS, U = ROWS / STEP;
  const int r = threadIdx.x % ROWS, cb = threadIdx.x / ROWS, k8 = (k + 7) & ~7;
  double x[U], dx[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int c = cb + STEP * u;
    const bool in = r < k && c < k;
    x[u] = in ? X[r + c * k] : (r == c ? 1.0 : 0.0);
    dx[u] = in ? dX[r + c * k] : 0.0;
  }
  for (int round = 0; round < seq; ++round) {
    __syncthreads();
    if (r < k8)
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (cb + STEP * u < k8) M[(cb + STEP * u) * FLD + r] = x[u] + *t * dx[u];
    double mn, mx;
    bool ok = cta_tile_chol(M, k, inv, sfail, &mn, &mx, red);
    if (ok && ratio > 0.0) ok = isfinite(mn) && isfinite(mx) && mx > 0 && mn > ratio * mx;
    if (ok || *t < min_step) return true;
    *t *= gamma;
  }
  return false;
}
constexpr int kTrialRounds = 4096;

// Orders above kSmallTrialOrder.  µs of a launch that takes 1, 2, 4 and 22 trials, eight at
// a time by warp_trial / this: 1 × order 48  154 153 154 441 / 12 19 37 154, 512 × order 48
// 344 346 344 1003 / 32 49 102 411, 512 × order 64 1199 1200 1198 3543 / 38 63 133 552.
__device__ double cta_backtrack(const double* X, const double* dX, int k, double gamma, double min_step,
                                double ratio, double* M, double* inv, int* sfail, double* red) {
  double t = 1.0;
  cta_trials<64>(X, dX, k, gamma, min_step, ratio, kTrialRounds, M, inv, sfail, red, &t);
  return t;
}

// Smaller orders: two trials like that (none up to order 8), which is as far as most
// searches go, then eight at a time, a warp each.  µs of a launch that takes 1, 2, 4 and
// 22 trials, all by the CTA / eight at a time by warp_trial / this:
//   1 × order 16     9 12 20 67      24 23 23 59      9 12 20 33
//   512 × order 8    15 22 44 166    20 20 20 44      16 15 15 28
//   512 × order 16   20 30 61 249    40 38 39 100     14 22 40 73
//   512 × order 32   26 44 97 413    122 122 120 337  20 30 80 173
// sm: a tile, or 10 packed slots of k(k+1)/2.
__device__ double cta_backtrack_small(const double* X, const double* dX, int k, double gamma, double min_step,
                                      double ratio, double* sm, double* inv, int* sfail, double* red, int* flags) {
  double t = 1.0;
  if (cta_trials<32>(X, dX, k, gamma, min_step, ratio, k <= 8 ? 0 : 2, sm, inv, sfail, red, &t)) return t;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, kp = k * (k + 1) / 2;
  double *Xp = sm, *dXp = sm + kp, *slot = sm + (2 + w) * kp;
  cta_load_packed(X, dX, k, Xp, dXp);
  for (int round = 0; round < kTrialRounds / kTrialWarps; ++round) {
    double cand[kTrialWarps], mine = 0.0;
#pragma unroll
    for (int j = 0; j < kTrialWarps; ++j) {
      cand[j] = j == 0 ? t : cand[j - 1] * gamma;
      if (j == w) mine = cand[j];
    }
    const bool ok = warp_trial_rows(Xp, dXp, mine, k, ratio, slot);
    if (lane == 0) flags[w] = ok;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kTrialWarps; ++j)
      if (flags[j] || cand[j] < min_step) return cand[j];
    t = cand[kTrialWarps - 1] * gamma;
    __syncthreads();  // the flags are read
  }
  return t;
}

// ------------------------------------- fraction to the boundary by eigenvalue
// X + t·dX = L(I + t·G)Lᵀ with G = L⁻¹·dX·L⁻ᵀ, so X + t·dX stays positive
// definite for t < t* = −1/λ_min(G) (every t when λ_min ≥ 0).  The bound is
// 1 when 1 + λ_min(G) > 0 (the full step stays interior), else t*: the value
// the bisection of `fraction_to_boundary_bound!` approaches from below, up to
// the rounding of its Cholesky tests.  λ_min comes from a Householder
// tridiagonalisation of G and a Sturm-count multisection of the tridiagonal
// matrix (one shift per thread per round).


// The bounds of both sides: the left half of the CTA takes X along dX, the right half
// Y along dY.  W = L_X⁻¹ and L_Y as left by the residual phase (global, k×k); S0, S1,
// S2: tiles.  out[0], out[1] (shared) receive the bounds.
__device__ __forceinline__ void cta_ftb_eig(const double* W, const double* LY, const double* dX,
                                            const double* dY, int k, double* S0, double* S1, double* S2,
                                            LambdaScratch* ls, double* inv, double* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nb = (k + 7) / 8;
  // M ← G = W·M·Wᵀ with Wt = Wᵀ in a tile, the strips' products W·M kept in registers.
  auto congruence = [&](const double* Wt, double* M) {
    double x[8][2] = {}, y[8][2] = {};
    if (warp < nb) {
      for (int p = 0; p < 2 * warp + 2; ++p) {  // W is lower
        const int q = 4 * p + t;
        const double a = Wt[(8 * warp + g) * FLD + q];
#pragma unroll
        for (int f = 0; f < 8; ++f)
          if (f < nb) tile64::mma8(x[f][0], x[f][1], a, M[(8 * f + g) * FLD + q]);
      }
#pragma unroll
      for (int p = 0; p < 16; ++p) {
        const int src = (lane & 28) | (2 * (p & 1) + (t >> 1)), q = 4 * p + t;
        const double v0 = __shfl_sync(0xffffffffu, x[p / 2][0], src);
        const double v1 = __shfl_sync(0xffffffffu, x[p / 2][1], src);
        const double a = (t & 1) ? v1 : v0;
#pragma unroll
        for (int f = p / 2; f < 8; ++f)  // Wᵀ is upper
          if (f < nb && p < 2 * nb) tile64::mma8(y[f][0], y[f][1], a, Wt[(8 * f + g) * FLD + q]);
      }
    }
    __syncthreads();
    if (warp < nb)
#pragma unroll
      for (int f = 0; f < 8; ++f)
        if (f < nb) {
          M[(8 * f + 2 * t) * FLD + 8 * warp + g] = y[f][0];
          M[(8 * f + 2 * t + 1) * FLD + 8 * warp + g] = y[f][1];
        }
  };
  cta_load_tile(S0, W, k, true);
  cta_load_tile(S1, dX, k);
  cta_load_tile(S2, LY, k);
  __syncthreads();
  if (threadIdx.x < 64 && (int)threadIdx.x < 8 * nb) inv[threadIdx.x] = 1.0 / S2[threadIdx.x * FLD + threadIdx.x];
  congruence(S0, S1);
  __syncthreads();
  cta_tile_inverse_t(S0, S2, inv, nb);  // S0 = L_Y⁻ᵀ
  cta_load_tile(S2, dY, k);
  __syncthreads();
  congruence(S0, S2);
  __syncthreads();
  for (int e = threadIdx.x; e < 64 * k; e += kThreads) {  // G and Gᵀ differ in rounding only
    const int r = e & 63, c = e >> 6;
    if (r < k && r > c) {
      S1[c * FLD + r] = S1[r * FLD + c] = 0.5 * (S1[c * FLD + r] + S1[r * FLD + c]);
      S2[c * FLD + r] = S2[r * FLD + c] = 0.5 * (S2[c * FLD + r] + S2[r * FLD + c]);
    }
  }
  __syncthreads();
  const int side = warp >> 2;
  const double b = lambda_bound_64(side ? S2 : S1, k, ls[side], (int)threadIdx.x & 127, 6 + side);
  if ((threadIdx.x & 127) == 0) out[side] = b;
  __syncthreads();
}

}  // namespace batch
}  // namespace sdpx
